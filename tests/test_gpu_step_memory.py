"""A context takes the band arrays with its others (three device allocations in
all, a batch five), and steps on the packed path, with the same bits, when they
cannot be had."""
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


@pytest.mark.parametrize("batch", [False, True])
def test_allocations_of_a_context_that_steps_in_bands(batch):
    import demso_b200 as D
    L = D.load()
    sc = scenes.agitated_gas(n=3000, seed=8, vel_std=1.0, pitch_factor=1.1, jitter=0.1)
    base = L.dem_debug_live_allocations()
    sim = D.Batch([(sc.sys, sc.n)]) if batch else D.Simulation(sc.sys, capacity=sc.n + 7)
    sim.set_state(*(_t(getattr(sc, k)) for k in FIELDS))
    sim.step(8)
    assert L.dem_debug_live_allocations() - base == (5 if batch else 3)
    got = sim.get_state("cpu")
    sim.close()
    assert L.dem_debug_live_allocations() == base
    ref = PortOracle("f32").run(sc.sys, sc.state(), 8)
    for k in ("pos", "vel", "theta", "omega", "pressure"):
        assert same(got[k].numpy(), ref[k]), k


def test_a_resident_scene_whose_band_arrays_cannot_be_had():
    # they are allocated after its cluster launches, at the call that would use them
    import demso_b200 as D
    L = D.load()
    sc = scenes.agitated_gas(n=2000, seed=9, vel_std=1.0, pitch_factor=1.1, jitter=0.1)
    sim = D.Simulation(sc.sys, capacity=sc.n, flags=D.CTX_PRESSURE | D.CTX_RESIDENT)
    sim.set_state(*(_t(getattr(sc, k)) for k in FIELDS))
    sim.step(512)
    try:
        D.check(L.dem_debug_fail_allocation(1))
        sim.step(8)
    finally:
        L.dem_debug_fail_allocation(0)
    sim.step(8)
    sim.check()
    got = sim.get_state("cpu")
    sim.close()
    ref = PortOracle("f32").run(sc.sys, sc.state(), 528)
    for k in ("pos", "vel", "theta", "omega", "pressure"):
        assert same(got[k].numpy(), ref[k]), k
