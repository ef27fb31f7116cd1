"""Short calls in a row leave the bands for the packed path, whose single steps
alternate between the two state sets (bands pack into the same one)."""
import numpy as np
import pytest

from demso_b200 import scenes
from helpers import same
from oracle.oracle import PortOracle

pytestmark = pytest.mark.gpu


def _t(a):
    import torch
    a = np.ascontiguousarray(a)
    return torch.from_numpy(a.view(np.int32).copy() if a.dtype == np.uint32 else a.copy())


@pytest.mark.parametrize("followed", [False, True])
def test_single_steps_after_a_longer_call(followed):
    import demso_b200 as D
    sc = scenes.agitated_gas(n=3000, seed=23, vel_std=2.0, pitch_factor=1.1, jitter=0.1)
    sim = D.Simulation(sc.sys, capacity=sc.n, flags=D.CTX_PRESSURE | D.CTX_ACCEL)
    sim.set_state(*(_t(getattr(sc, k)) for k in ("pos", "vel", "theta", "omega", "radius", "mass",
                                                 "id")))
    before = sim.state_view()["set"]
    sim.step(8)
    # 15 single steps in bands, 16 on the packed path and, to be read off, one
    # more there
    rows = []
    for _ in range(32):
        if followed:
            rows.append(sim.step_followed(1, [0, 1234, 2999])[0])
        else:
            sim.step(1)
    assert sim.state_view()["set"] != before
    got = {k: v.numpy() for k, v in sim.get_state("cpu").items() if v is not None}
    sim.check()
    sim.close()
    ref = PortOracle("f32")
    r = ref.run(sc.sys, sc.state(), 40)
    for k in ("pos", "vel", "theta", "omega", "pressure", "acc", "alpha"):
        assert same(got[k], r[k]), k
    for k in (0, 14, 15, 16, 31) if followed else ():
        r = ref.run(sc.sys, sc.state(), 9 + k)
        for j, i in enumerate((0, 1234, 2999)):
            assert same(rows[k][j, 2:4], r["pos"][r["loc"][i]]), (k, i)
            assert same(rows[k][j, 11], r["pressure"][r["loc"][i]]), (k, i)
