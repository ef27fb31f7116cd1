"""The gradient does not depend on how many steps a window of the reverse pass
re-runs, nor on the path they take: one step (packed), several (bands), all of
them, crowded cells (packed)."""
import numpy as np
import pytest

from demso_b200 import scenes

pytestmark = pytest.mark.gpu


def _t(a):
    import torch
    a = np.ascontiguousarray(a)
    return torch.from_numpy(a.view(np.int32).copy() if a.dtype == np.uint32 else a.copy())


@pytest.mark.parametrize("kind", ["scene", "batch", "crowded"])
def test_windows_of_any_length(kind):
    import torch
    import demso_b200 as D
    flags = D.CTX_PRESSURE | D.CTX_ACCEL
    if kind == "batch":
        parts = [scenes.agitated_gas(n=n, seed=n, vel_std=2.0, pitch_factor=1.1, jitter=0.1)
                 for n in (700, 60, 1500)]
        st, sim = scenes.concat_specimens(parts), D.Batch([(p.sys, p.n) for p in parts], flags)
    else:
        n, grid = (40000, (32, 16)) if kind == "crowded" else (2000, "2r")
        sc = scenes.agitated_gas(n=n, seed=4, vel_std=2.0, grid=grid, pitch_factor=1.1, jitter=0.1)
        st, sim = sc.state(), D.Simulation(sc.sys, capacity=sc.n, flags=flags)
    n = st["pos"].shape[0]
    rng = np.random.default_rng(0)
    lam0 = [rng.normal(size=s).astype(np.float32) for s in ((n, 2), (n, 2), (n,))]
    out = []
    for every in (1, 2, 5, 11):
        sim.set_state(*(_t(st[k]) for k in ("pos", "vel", "theta", "omega", "radius", "mass",
                                            "id")))
        lam = [_t(x).cuda() for x in lam0]
        sim.adjoint_forward(11, every)
        grad = sim.adjoint_backward(*lam)
        sim.check()
        out.append([x.cpu().numpy() for x in lam] + [grad])
    sim.close()
    assert np.any(out[0][3] != 0)
    for o in out[1:]:
        for a, b in zip(out[0], o):
            assert np.array_equal(a, b)
