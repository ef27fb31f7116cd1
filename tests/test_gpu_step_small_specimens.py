"""Batches of specimens of a single band (no free slots) and of several, few and
many movers, more events than a band takes: the oracle's bits for each."""
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


@pytest.mark.parametrize("counts,vel", [((1, 2, 31, 33, 28, 28), 3.0), ((900, 1, 700), 60.0),
                                        ((28, 3000, 1, 5000, 60), 3.0), ((800, 800), 300.0),
                                        ((40, 3000, 40), 100.0)])
def test_specimens_of_one_band_and_of_several(counts, vel):
    import torch
    import demso_b200 as D
    parts = [scenes.agitated_gas(n=n, seed=40 + k, vel_std=vel, n_mat=1 + k % 2, pitch_factor=1.1,
                                 jitter=0.1) for k, n in enumerate(counts)]
    st = scenes.concat_specimens(parts)
    sim = D.Batch([(p.sys, p.n) for p in parts], flags=D.CTX_PRESSURE | D.CTX_ACCEL)
    fields = ("pos", "vel", "theta", "omega", "radius", "mass", "id", "type")
    sim.set_state(*(_t(st[k]) for k in fields))
    for k in (5, 1, 24):
        sim.step(k)
    torch.cuda.synchronize()
    sim.check()
    got = {k: v.numpy() for k, v in sim.get_state("cpu").items() if v is not None}
    sim.close()
    a = 0
    for p in parts:
        s = p.state()
        if s.get("type") is None:
            s["type"] = np.zeros(p.n, np.uint32)
        ref = PortOracle("f32").run(p.sys, s, 30)
        for k in ("pos", "vel", "theta", "omega", "pressure", "acc", "alpha"):
            assert same(got[k][a:a + p.n], ref[k]), (p.n, k)
        assert np.array_equal(got["id"].view(np.uint32)[a:a + p.n] - a, ref["id"]), p.n
        a += p.n
