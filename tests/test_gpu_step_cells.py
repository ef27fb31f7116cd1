"""Cell ranges and row slots describe the sort of the last step, whatever has
replaced the parameters or the state since: asked for after new parameters
(dem_set_system, dem_batch_set_systems) or a new state, they are those of a
twin that was asked before."""
import copy
import ctypes as C

import numpy as np
import pytest

from demso_b200 import scenes

pytestmark = pytest.mark.gpu


def _t(a):
    import torch
    a = np.ascontiguousarray(a)
    return torch.from_numpy(a.view(np.int32).copy() if a.dtype == np.uint32 else a.copy())


def _load(sim, st):
    sim.set_state(*(_t(st[k]) for k in ("pos", "vel", "theta", "omega", "radius", "mass", "id")))


def _cells(sim, cells):
    import torch
    import demso_b200 as D
    cs, ce = (torch.empty(cells, dtype=torch.int32, device="cuda") for _ in range(2))
    D.check(D.load().dem_get_cells(sim.handle, cs.data_ptr(), ce.data_ptr(), D._stream()))
    cs, ce = cs.cpu().numpy().view(np.uint32), ce.cpu().numpy().view(np.uint32)
    return cs, np.where(cs == 0xFFFFFFFF, 0, ce)


def _rows(sim, lo, hi):
    import demso_b200 as D
    a, b = C.c_uint32(), C.c_uint32()
    D.check(D.load().dem_row_slots(sim.handle, lo, hi, C.byref(a), C.byref(b), D._stream()))
    return a.value, b.value


def _changed(sys):
    s = copy.deepcopy(sys)
    s.Lx, s.Ly, s.dt = 1.1 * s.Lx, 1.2 * s.Ly, 0.5 * s.dt
    return s


def _asked(make, steps, change, ask):
    """(answer asked before the change, answer asked after it)."""
    out = []
    for first in (True, False):
        sim = make()
        for k in steps:
            sim.step(k)
        if first:
            out.append(ask(sim))
        else:
            change(sim)
            out.append(ask(sim))
        sim.close()
    return out


def _equal(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("steps", [(20,), (2, 20), (20, 3)])
@pytest.mark.parametrize("rows", [None, (8, 32)])
def test_after_new_parameters(rows, steps):
    import demso_b200 as D
    sc = scenes.agitated_gas(n=4096, seed=3, vel_std=3.0, grid=(32, 64), pitch_factor=1.1,
                             jitter=0.1)
    st = sc.state()
    if rows:
        from demso_b200.slab import cell_rows
        r = cell_rows(sc.sys, sc.pos)
        at = np.nonzero((r >= rows[0] + 4) & (r < rows[0] + rows[1] - 4))[0]
        st = {k: (v[at].copy() if v is not None else None) for k, v in st.items()}
        st["id"] = np.arange(at.size, dtype=np.uint32)
    nrows = rows[1] if rows else sc.sys.gy
    lo = rows[0] if rows else 0

    def make():
        sim = D.Simulation(sc.sys, capacity=st["pos"].shape[0], rows=rows)
        _load(sim, st)
        return sim

    ask = lambda sim: _cells(sim, sc.sys.gx * nrows) + (_rows(sim, lo + 5, lo + 11),)
    a, b = _asked(make, steps, lambda sim: sim.set_system(_changed(sc.sys)), ask)
    assert np.count_nonzero(a[0] != 0xFFFFFFFF) > 100
    assert _equal(a, b)
    # the cells of a new state's predecessor, as far as dem_get_cells goes
    ask = lambda sim: _cells(sim, sc.sys.gx * nrows)
    a, b = _asked(make, steps, lambda sim: _load(sim, st), ask)
    assert _equal(a, b)


@pytest.mark.parametrize("steps", [(20,), (1, 20), (20, 2)])
def test_after_new_parameters_of_a_batch(steps):
    import demso_b200 as D
    parts = [scenes.agitated_gas(n=n, seed=n, vel_std=3.0, pitch_factor=1.1, jitter=0.1)
             for n in (300, 2500, 40)]
    st = scenes.concat_specimens(parts)

    def make():
        sim = D.Batch([(p.sys, p.n) for p in parts])
        _load(sim, st)
        return sim

    cells = sum(p.sys.num_cells for p in parts)
    a, b = _asked(make, steps, lambda sim: sim.set_systems([_changed(p.sys) for p in parts]),
                  lambda sim: _cells(sim, cells))
    assert np.count_nonzero(a[0] != 0xFFFFFFFF) > 100
    assert _equal(a, b)


def test_cells_of_a_batch():
    # the arrays hold every specimen's cells, not the first one's
    import demso_b200 as D
    parts = [scenes.agitated_gas(n=n, seed=n, vel_std=3.0, pitch_factor=1.1, jitter=0.1)
             for n in (300, 2500, 40)]
    sim = D.Batch([(p.sys, p.n) for p in parts])
    _load(sim, scenes.concat_specimens(parts))
    sim.step(5)
    cs, ce = (x.cpu().numpy().view(np.uint32) for x in sim.cells())
    n = sum(p.sys.num_cells for p in parts)
    assert cs.size == ce.size == n
    want = _cells(sim, n)
    assert np.array_equal(cs, want[0])
    assert np.array_equal(np.where(cs == 0xFFFFFFFF, 0, ce), want[1])
    assert int((want[1] - np.where(cs == 0xFFFFFFFF, 0, cs)).sum()) == 2840
    sim.close()
