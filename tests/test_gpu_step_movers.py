"""Scenes in which many disks change cell step on the packed path, others in
bands, at a new state and as a scene speeds up or slows down; the bits are the
oracle's throughout.  A call of an odd number of packed steps leaves the state
in the other of the two sets (bands pack into the same one)."""
import copy

import numpy as np
import pytest

from demso_b200 import scenes
from helpers import same
from oracle.oracle import PortOracle

pytestmark = pytest.mark.gpu

FIELDS = ("pos", "vel", "theta", "omega", "radius", "mass", "id")


def _t(a):
    import torch
    a = np.ascontiguousarray(a)
    return torch.from_numpy(a.view(np.int32).copy() if a.dtype == np.uint32 else a.copy())


def _load(sim, st):
    sim.set_state(*(_t(st[k]) for k in FIELDS))


def _call(sim, steps):
    """Whether an odd call took packed steps."""
    import torch
    assert steps & 1
    before = sim.state_view()["set"]
    sim.step(steps)
    torch.cuda.synchronize()  # what the call reports has arrived
    return sim.state_view()["set"] != before


def _same(sim, ref):
    got = sim.get_state("cpu")
    sim.check()
    for k in ("pos", "vel", "theta", "omega", "pressure"):
        assert same(got[k].numpy(), ref[k]), k


def _gas(grid, n, vel, seed=5, jit=0.2):
    """n disks spread over all rows of a grid of 2.2 mm cells."""
    sc = scenes.agitated_gas(n=n, seed=seed, vel_std=vel, grid=grid, gravity=(0.0, 0.0))
    sc.sys.Lx, sc.sys.Ly = grid[0] * 2.2e-3, grid[1] * 2.2e-3
    nx = int(np.ceil(np.sqrt(n * grid[0] / grid[1])))
    ny = -(-n // nx)
    k = np.arange(n)
    rng = np.random.default_rng(seed)
    sc.pos[:] = (np.stack([k % nx, k // nx], 1) + rng.uniform(0.5 - jit, 0.5 + jit, (n, 2))) * \
        [sc.sys.Lx / nx, sc.sys.Ly / ny]
    return sc


# 512 bands (one row each) and 256 (whose limit is the free slots)
@pytest.mark.parametrize("grid,fast,slow", [((512, 512), 150.0, 2.0), ((256, 256), 400.0, 20.0)])
def test_new_states_and_scenes_that_change(grid, fast, slow):
    import demso_b200 as D
    sc = _gas(grid, 20000, 1.0, jit=0.35) if grid[0] == 512 else _gas(grid, 30000, 1.0)
    ref = PortOracle("f32")
    sim = D.Simulation(sc.sys, capacity=sc.n)
    st = sc.state()
    unit = st["vel"].copy()

    def go(speed):
        st["vel"] = (unit * np.float32(speed)).astype(np.float32)
        _load(sim, st)

    go(slow)
    sim.step(512)  # long enough for calls to report
    for speed, packed in ((slow, False), (fast, True), (slow, False)):
        go(speed)
        assert _call(sim, 7) == packed
        _same(sim, ref.run(sc.sys, st, 7))
    # the scene speeds up: the call that finds out is in bands, the next is not
    v = sim.state_view()
    v["vel"].mul_(fast / slow)
    assert not _call(sim, 21)
    assert _call(sim, 21)
    # and slows down: after 512 packed steps (the second wait) an estimate, then bands
    sim.state_view()["vel"].mul_(1e-3)
    assert _call(sim, 511)
    assert _call(sim, 1)
    assert not _call(sim, 21)
    b = ref.run(sc.sys, st, 7)
    b["vel"] = (b["vel"] * np.float32(fast / slow)).astype(np.float32)
    b = ref.run(sc.sys, b, 42)
    b["vel"] = (b["vel"] * np.float32(1e-3)).astype(np.float32)
    _same(sim, ref.run(sc.sys, b, 533))
    sim.close()


def test_followed_rows_and_a_batch_with_many_movers():
    import demso_b200 as D
    sc = _gas((512, 512), 20000, 150.0, jit=0.35)
    ref = PortOracle("f32")
    sim = D.Simulation(sc.sys, capacity=sc.n)
    _load(sim, sc.state())
    rows = sim.step_followed(9, [0, 19999])
    _same(sim, ref.run(sc.sys, sc.state(), 9))
    for k in (0, 8):
        r = ref.run(sc.sys, sc.state(), k + 1)
        for j, i in enumerate((0, 19999)):
            assert same(rows[k, j, 2:4], r["pos"][r["loc"][i]])
    sim.close()
    # 320 specimens of one band each
    parts = [_gas((16, 16), 60, 200.0, seed=k) for k in range(320)]
    st = scenes.concat_specimens(parts)
    sim = D.Batch([(p.sys, p.n) for p in parts])
    _load(sim, st)
    assert _call(sim, 9)
    got = sim.get_state("cpu")
    sim.check()
    sim.close()
    for k in (0, 1, 319):
        r = ref.run(parts[k].sys, parts[k].state(), 9)
        for x in ("pos", "vel", "theta", "omega", "pressure"):
            assert same(got[x].numpy()[60 * k:60 * k + 60], r[x]), x


@pytest.mark.parametrize("n,grid,packed", [(40000, (32, 16), True), (22000, (16, 8), True),
                                           (20000, (32, 16), False), (2000, (16, 4), False)])
def test_crowded_cells(n, grid, packed):
    # rows of 234, 515, 117 and 94 candidates; 9.4, 11, 2.3 and 0.2 million of them
    import demso_b200 as D
    sc = scenes.agitated_gas(n=n, seed=3, vel_std=0.5, grid=grid, pitch_factor=1.1, jitter=0.1)
    sim = D.Simulation(sc.sys, capacity=n)
    _load(sim, sc.state())
    assert _call(sim, 5) == packed
    _same(sim, PortOracle("f32").run(sc.sys, sc.state(), 5))
    sim.close()


@pytest.mark.parametrize("crowd,packed", [(30000, True), (9000, False)])
def test_crowded_specimens(crowd, packed):
    # the crowded specimen's tests decide (10.5 and 0.95 million), not the average
    import demso_b200 as D
    parts = [scenes.agitated_gas(n=crowd, seed=3, vel_std=0.5, grid=(16, 16), pitch_factor=1.1,
                                 jitter=0.1),
             scenes.agitated_gas(n=300, seed=4, vel_std=0.5, grid=(512, 256), box=1.0)]
    st = scenes.concat_specimens(parts)
    sim = D.Batch([(p.sys, p.n) for p in parts])
    _load(sim, st)
    assert _call(sim, 5) == packed
    got = sim.get_state("cpu")
    sim.check()
    sim.close()
    ref = PortOracle("f32").run(parts[0].sys, parts[0].state(), 5)
    for x in ("pos", "vel", "theta", "omega", "pressure"):
        assert same(got[x].numpy()[:crowd], ref[x]), x


@pytest.mark.parametrize("crowded", [False, True])
def test_a_resident_batch(crowded):
    # with many movers it is packed (single steps alternate the sets), with crowded
    # cells its calls of three steps or more are resident launches
    import demso_b200 as D
    if crowded:
        parts = [scenes.agitated_gas(n=6000, seed=k, vel_std=0.5, grid=(8, 8), pitch_factor=1.1,
                                     jitter=0.1) for k in range(6)]
    else:
        parts = [_gas((16, 16), 60, 200.0, seed=k) for k in range(320)]
    st = scenes.concat_specimens(parts)
    sim = D.Batch([(p.sys, p.n) for p in parts], flags=D.CTX_PRESSURE | D.CTX_RESIDENT)
    _load(sim, st)
    assert _call(sim, 9) != crowded
    assert _call(sim, 1)
    sim.step(2)
    sim.step(4)
    got = sim.get_state("cpu")
    sim.check()
    sim.close()
    n = parts[0].n
    for k in (0, 3, len(parts) - 1):
        r = PortOracle("f32").run(parts[k].sys, parts[k].state(), 16)
        for x in ("pos", "vel", "theta", "omega", "pressure"):
            assert same(got[x].numpy()[n * k:n * k + n], r[x]), x


@pytest.mark.parametrize("vel,packed", [(0.5, False), (20.0, True)])
def test_a_state_looked_at_in_part(vel, packed):
    # 2.2 million disks in 1,024 bands: every second block of 256; about 0.8 and 31
    # movers a band
    import demso_b200 as D
    sc = scenes.agitated_gas(n=2200000, seed=6, vel_std=vel, pitch_factor=1.5, jitter=0.1,
                             gravity=(0.0, 0.0))
    sim = D.Simulation(sc.sys, capacity=sc.n)
    _load(sim, sc.state())
    assert _call(sim, 5) == packed
    _same(sim, PortOracle("f32").run(sc.sys, sc.state(), 5))
    sim.close()
