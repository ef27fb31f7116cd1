"""dem_set_state and dem_get_state with device arrays: the one-launch copy, and
arrays it does not take (odd addresses), give the arrays of host copies."""
import numpy as np
import pytest

from demso_b200 import scenes
from helpers import same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 5, 1023, 70001])
@pytest.mark.parametrize("shift", [0, 1])
def test_device_copies_equal_host_copies(n, shift):
    import torch
    import demso_b200 as D
    sc = scenes.agitated_gas(n=n, seed=n, n_mat=2, grid=(64, 64), box=0.6)
    t = lambda a: torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a)

    def moved(a):
        # `shift` elements past a 16-byte boundary (8 bytes for pairs, 4 for words)
        h = t(a)
        d = torch.empty(h.numel() + 2 * shift * max(1, h[0].numel()), dtype=h.dtype, device="cuda")
        d = d[shift * max(1, h[0].numel()):][:h.numel()].view(h.shape)
        return d.copy_(h)

    out = {}
    for where, f in (("host", t), ("device", moved)):
        sim = D.Simulation(sc.sys, capacity=n, flags=D.CTX_PRESSURE | D.CTX_ACCEL)
        sim.set_state(*(f(a) for a in (sc.pos, sc.vel, sc.theta, sc.omega, sc.radius, sc.mass,
                                       sc.id, sc.type)))
        if where == "device":
            torch.cuda.synchronize()
        sim.step(3)
        out[where] = {k: v.cpu().numpy() for k, v in
                      sim.get_state("cpu" if where == "host" else "cuda").items()}
        sim.close()
    for k in out["host"]:
        assert same(out["host"][k], out["device"][k]), k
