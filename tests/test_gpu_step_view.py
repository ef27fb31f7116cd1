"""What is written through the state view between two calls is part of the
next step, whichever path made the state and takes the step."""
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


@pytest.mark.parametrize("calls", [(8, 8), (20, 1), (1, 8), (2, 2), (5, 3, 9)])
def test_edits_through_the_view(calls):
    import torch
    import demso_b200 as D
    sc = scenes.agitated_gas(n=5000, seed=17, vel_std=2.0, n_mat=2, pitch_factor=1.1, jitter=0.1)
    sim = D.Simulation(sc.sys, capacity=sc.n, flags=D.CTX_PRESSURE | D.CTX_ACCEL)
    st = sc.state()
    sim.set_state(*(_t(st[k]) for k in ("pos", "vel", "theta", "omega", "radius", "mass", "id",
                                        "type")))
    ref = PortOracle("f32")
    for k, n in enumerate(calls):
        if k:
            v = sim.state_view()
            v["vel"].mul_(0.5)
            v["omega"].add_(3.0)
            v["mass"].mul_(1.25)
            st["vel"] = (st["vel"] * np.float32(0.5)).astype(np.float32)
            st["omega"] = (st["omega"] + np.float32(3.0)).astype(np.float32)
            st["mass"] = (st["mass"] * np.float32(1.25)).astype(np.float32)
        sim.step(n)
        st = ref.run(sc.sys, st, n)
    got = sim.get_state("cpu")
    torch.cuda.synchronize()
    sim.check()
    sim.close()
    for k in ("pos", "vel", "theta", "omega", "mass", "pressure", "acc", "alpha"):
        assert same(got[k].numpy(), st[k]), k
    assert np.array_equal(got["id"].numpy().view(np.uint32), st["id"])
