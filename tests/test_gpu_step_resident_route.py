"""Which calls of a resident scene of more than 1,536 disks are cluster launches:
the first 160 steps, then short calls that are not in bands.
After a cluster launch the state is in no sort's order (dem_row_slots refuses),
after the graph path it is.  The bits are the same on both."""
import ctypes as C

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


def _by_cluster(sim):
    import demso_b200 as D
    a, b = C.c_uint32(), C.c_uint32()
    return D.load().dem_row_slots(sim.handle, 0, 1, C.byref(a), C.byref(b), D._stream()) != 0


@pytest.mark.parametrize("n,short", [(1600, [False, True, True, True, False]),
                                     (3500, [False, False, True, False, False]),
                                     (7000, [False, False, False, False, False])])
def test_calls_of_a_resident_scene(n, short):
    import demso_b200 as D
    sc = scenes.agitated_gas(n=n, seed=n, vel_std=1.0, pitch_factor=1.1, jitter=0.1)
    sim = D.Simulation(sc.sys, capacity=n, flags=D.CTX_PRESSURE | D.CTX_RESIDENT)
    load = lambda: sim.set_state(*(_t(getattr(sc, k)) for k in FIELDS))
    load()
    sim.step(3)
    assert _by_cluster(sim)
    sim.step(100)
    assert _by_cluster(sim)
    sim.step(57)
    assert _by_cluster(sim)
    sim.step(8)  # the 161st step
    assert not _by_cluster(sim)
    sim.step(2)  # stays in the bands
    assert not _by_cluster(sim)
    sim.check()
    got = sim.get_state("cpu")
    ref = PortOracle("f32").run(sc.sys, sc.state(), 170)
    for k in ("pos", "vel", "theta", "omega", "pressure"):
        assert same(got[k].numpy(), ref[k]), k
    for steps, cluster in zip((1, 2, 3, 7, 8), short):
        load()  # not in bands
        sim.step(steps)
        assert _by_cluster(sim) == cluster, steps
        got = sim.get_state("cpu")
        ref = PortOracle("f32").run(sc.sys, sc.state(), steps)
        for k in ("pos", "vel", "theta", "omega", "pressure"):
            assert same(got[k].numpy(), ref[k]), (steps, k)
    sim.close()
