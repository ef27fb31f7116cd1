"""The step in bands of cell rows with free slots: new layouts, bands that grow
and shrink, odd step counts and calls of other kinds in between, bit for bit
against the CPU restatement of the reference."""
import numpy as np
import pytest

from demso_b200 import scenes
from helpers import EMPTY, gpu_run, occupied_cell_end, same
from oracle.oracle import PortOracle

pytestmark = pytest.mark.gpu

KEYS = ("pos", "vel", "theta", "omega", "pressure", "acc", "alpha", "id", "loc")


def _check(sc, steps, chunks=None):
    got = gpu_run(sc.sys, sc.state(), steps, chunks=chunks)
    ref = PortOracle("f32").run(sc.sys, sc.state(), steps)
    for k in KEYS:
        assert same(got[k], ref[k]), k


@pytest.mark.parametrize("grid", [(1, 1), (2, 2), (64, 4), (4, 64), (256, 2), (4096, 1),
                                  (8192, 1)])
def test_grids_of_one_band_many_bands_and_wide_rows(grid):
    # 1 band (up to 256 cells), bands of several rows, of one row, the widest
    # row of a band, and a wider one (the packed path); the box is wide enough
    # for cells of 2 rmax along the wide axis
    gx, gy = grid
    n = 700
    sc = scenes.agitated_gas(n=n, seed=3, vel_std=2.0, grid=grid, pitch_factor=1.1, jitter=0.1,
                             box=0.0583)
    if gx > 16:
        sc.sys.Lx = gx * 2.5e-3
    if gy > 16:
        sc.sys.Ly = gy * 2.5e-3
    _check(sc, 23, [1, 2, 3, 17])


@pytest.mark.parametrize("vel", [0.5, 20.0, 300.0])
@pytest.mark.parametrize("n_mat", [1, 3])
def test_few_movers_many_movers_and_overflowing_bands(vel, n_mat):
    # 300 m/s: a quarter of the disks change cell on every step, more than a
    # band's events, so every step lays the bands out again
    sc = scenes.agitated_gas(n=9001, seed=7, vel_std=vel, n_mat=n_mat, pitch_factor=1.15,
                             jitter=0.05)
    _check(sc, 41, [1, 1, 39])


def test_a_band_fills_up_and_empties():
    # everything falls into the lowest rows: their bands run out of free slots
    # and the layout is made again; upper bands run empty
    sc = scenes.agitated_gas(n=3000, seed=9, vel_std=0.1, pitch_factor=1.6, jitter=0.05,
                             gravity=(0.0, -2.0e5))
    sc.vel[:, 1] = -60.0
    _check(sc, 300)


def test_calls_of_other_kinds_between_calls():
    import torch
    import demso_b200 as D
    sc = scenes.agitated_gas(n=5000, seed=21, vel_std=3.0, pitch_factor=1.1, jitter=0.1)
    t = lambda a: torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a)
    ref = PortOracle("f32")

    def state(sim):
        return {k: (v.numpy().view(np.uint32) if k in ("id", "loc") else v.numpy())
                for k, v in sim.get_state("cpu").items() if v is not None}

    sim = D.Simulation(sc.sys, capacity=sc.n + 100, flags=D.CTX_PRESSURE | D.CTX_ACCEL)
    sim.set_state(t(sc.pos), t(sc.vel), t(sc.theta), t(sc.omega), t(sc.radius), t(sc.mass),
                  t(sc.id))
    sim.step(7)
    rows = sim.step_followed(8, [0, 17, 4999])
    cs, ce = (a.cpu().numpy().view(np.uint32) for a in sim.cells())
    first, count = sim_rows(sim, 3, 9)
    got = state(sim)
    r15 = ref.run(sc.sys, sc.state(), 15)
    for k in KEYS:
        assert same(got[k], r15[k]), k
    # the cells of the last sort, which ordered the positions before the last step
    r14 = ref.run(sc.sys, sc.state(), 14)
    by_id = np.empty((sc.n, 2), np.float32)
    by_id[r14["id"]] = r14["pos"]
    h = scenes.cell_hash(by_id[got["id"]], sc.sys)
    assert np.array_equal(np.sort(h), h)
    gx = sc.sys.gx
    assert (first, count) == (int(np.sum(h < 3 * gx)), int(np.sum((h >= 3 * gx) & (h < 9 * gx))))
    occ, start, num = np.unique(h, return_index=True, return_counts=True)
    assert np.array_equal(np.nonzero(cs != EMPTY)[0], occ)
    assert np.array_equal(cs[occ], start)
    assert np.array_equal(occupied_cell_end(cs, ce)[occ], start + num)
    for k in range(8):
        r = ref.run(sc.sys, sc.state(), 8 + k)
        for j, i in enumerate((0, 17, 4999)):
            at = r["loc"][i]
            assert same(rows[k, j, 2:4], r["pos"][at]) and same(rows[k, j, 11], r["pressure"][at])
    # the packed path (a control particle out of reach), then bands again
    sim.set_control((-5.0, -5.0), 1e-3)
    sim.step(6)
    sim.set_control(None, 0)
    sim.step(5)
    # the tuner and single steps
    sim.set_step_variant(2)
    for _ in range(3):
        sim.step(1)
    got = state(sim)
    r29 = ref.run(sc.sys, sc.state(), 29)
    for k in ("pos", "vel", "theta", "omega", "id"):
        assert same(got[k], r29[k]), k
    # fewer disks in the same context
    m = 1234
    sim.set_state(t(sc.pos[:m].copy()), t(sc.vel[:m].copy()), t(sc.theta[:m].copy()),
                  t(sc.omega[:m].copy()), t(sc.radius[:m].copy()), t(sc.mass[:m].copy()),
                  t(sc.id[:m].copy()))
    sim.step(12)
    sim.check()
    got = state(sim)
    sim.close()
    small = {k: (v[:m] if v is not None else None) for k, v in sc.state().items()}
    r12 = ref.run(sc.sys, small, 12)
    for k in KEYS:
        assert same(got[k], r12[k]), k


def sim_rows(sim, lo, hi):
    import ctypes as C
    import demso_b200 as D
    a, b = C.c_uint32(), C.c_uint32()
    D.check(D.load().dem_row_slots(sim.handle, lo, hi, C.byref(a), C.byref(b), D._stream()))
    return a.value, b.value


def test_cells_entered_in_steps_after_each_other():
    # more disks than the GPU has threads, so blocks of a step end before others
    # of it begin; every other disk sits at the edge of two cells, so disks change
    # cell in one step and in the next near each other, the rows beside the grid's
    # wrap included (first and last blocks)
    nx, ny = 8192, 64
    sc = scenes.agitated_gas(n=nx * ny, seed=5, vel_std=0.5, grid=(4096, 32))
    pitch = 2.05e-3
    rng = np.random.default_rng(5)
    ij = np.stack(np.meshgrid(np.arange(nx), np.arange(ny) + 0.5, indexing="xy"), -1)
    at = (ij.reshape(-1, 2) + rng.uniform(-0.025, 0.025, size=(nx * ny, 2))) * pitch
    sc.pos[:] = np.maximum(at, 1e-5)
    sc.sys.Lx, sc.sys.Ly = nx * pitch, ny * pitch
    # soft contacts: disks this slow search every few steps
    m = sc.sys.materials[0]
    m.normalStiffness, m.shearStiffness = 1e3, 5e2
    sc.sys.knWall, sc.sys.ktWall = 1e3, 5e2
    _check(sc, 40)


def test_disks_that_leave_a_row_window():
    # they are met across the window's wrap, from the last band to the first; calls
    # of 3 steps stay on the packed path
    from demso_b200.slab import cell_rows
    sc = scenes.agitated_gas(n=4096, seed=11, vel_std=0.5, grid=(64, 64), pitch_factor=1.15,
                             gravity=(0.0, 0.0))
    sc.pos[:, 1] = np.minimum(sc.pos[:, 1] + 1.15e-3, sc.sys.Ly - 1e-5)
    rows = (16, 32)
    r = cell_rows(sc.sys, sc.pos)
    at = np.nonzero((r >= rows[0]) & (r < rows[0] + rows[1]))[0]
    st = {k: (v[at].copy() if v is not None else None) for k, v in sc.state().items()}
    st["id"] = np.arange(at.size, dtype=np.uint32)
    a = gpu_run(sc.sys, st, 200, rows=rows)
    b = gpu_run(sc.sys, st, 200, rows=rows, chunks=[3] * 66 + [2])
    r = cell_rows(sc.sys, a["pos"])
    assert np.any((r < rows[0]) | (r >= rows[0] + rows[1]))
    for k in KEYS:
        assert same(a[k], b[k]), k


@pytest.mark.parametrize("n", [1220000, 1250000])
def test_sizes_beside_the_ten_block_shape(n):
    # 1,296,250 and 1,328,125 slots: the last of the 8-block shape, the first of
    # the 10-block one (from 1,310,720 on)
    sc = scenes.agitated_gas(n=n, seed=31, vel_std=2.0, pitch_factor=1.1, jitter=0.1)
    _check(sc, 8)


@pytest.mark.parametrize("kind", ["typed", "batch"])
def test_the_ten_block_shape_of_types_and_batches(kind):
    import torch
    import demso_b200 as D
    t = lambda a: torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a)
    if kind == "typed":
        sc = scenes.agitated_gas(n=1400000, seed=33, vel_std=2.0, pitch_factor=1.1, jitter=0.1,
                                 n_mat=3)
        st = sc.state()
        make = lambda: D.Simulation(sc.sys, capacity=sc.n, flags=D.CTX_PRESSURE | D.CTX_ACCEL)
    else:
        parts = [scenes.agitated_gas(n=n, seed=34 + n % 7, vel_std=2.0, pitch_factor=1.1,
                                     jitter=0.1) for n in (700001, 699, 701003)]
        st = scenes.concat_specimens(parts)
        make = lambda: D.Batch([(p.sys, p.n) for p in parts],
                               flags=D.CTX_PRESSURE | D.CTX_ACCEL)
    got = []
    for variant in (0, 1):  # 1 is one shape for every size
        sim = make()
        sim.set_step_variant(variant)
        sim.set_state(*(t(st[k]) for k in ("pos", "vel", "theta", "omega", "radius", "mass",
                                           "id")),
                      *([t(st["type"])] if kind == "typed" else []))
        sim.step(12)
        got.append({k: v.numpy() for k, v in sim.get_state("cpu").items() if v is not None})
        sim.check()
        sim.close()
    for k in got[0]:
        assert same(got[0][k], got[1][k]), k
