"""A sort whose bounded wait gives up while the context steps in bands (calls of
several steps): every access stays in bounds, the calls return, dem_check
reports the timeout, and after a new state the steps are the oracle's again."""
import numpy as np
import pytest

from demso_b200 import scenes
from helpers import same
from oracle.oracle import PortOracle

pytestmark = pytest.mark.gpu

TIMEOUT = 4
NO_HOLD = 0xFFFFFFFF
FIELDS = ("pos", "vel", "theta", "omega", "radius", "mass", "id", "type")


def _t(a):
    import torch
    a = np.ascontiguousarray(a)
    return torch.from_numpy(a.view(np.int32).copy() if a.dtype == np.uint32 else a.copy())


@pytest.mark.parametrize("tile", [0, 2])
@pytest.mark.parametrize("kind", ["plain", "attracting", "batch", "control", "adjoint"])
def test_bands_survive_a_sort_that_gives_up(kind, tile):
    import torch
    import demso_b200 as D
    L = D.load()
    flags = D.CTX_PRESSURE | D.CTX_ACCEL
    if kind == "batch":
        parts = [scenes.agitated_gas(n=n, seed=n, vel_std=2.0, pitch_factor=1.1, jitter=0.1)
                 for n in (9000, 500, 10500)]
        st = scenes.concat_specimens(parts)
        sim = D.Batch([(p.sys, p.n) for p in parts], flags=flags)
    else:
        sc = scenes.agitated_gas(n=20000, seed=81, vel_std=2.0, pitch_factor=1.1, jitter=0.1,
                                 n_mat=3 if kind == "attracting" else 1,
                                 attraction=20.0 if kind == "attracting" else 0.0)
        parts, st = [sc], sc.state()
        sim = D.Simulation(sc.sys, capacity=sc.n, flags=flags)
    n = st["pos"].shape[0]
    load = lambda: sim.set_state(*(_t(st[k]) for k in FIELDS if st.get(k) is not None))
    ids = np.arange(0, n, 97)

    def gave_up():
        torch.cuda.synchronize()
        with pytest.raises(D.DemError) as e:
            sim.check()
        assert e.value.code == TIMEOUT

    D.check(L.dem_debug_sort_hold(sim.handle, tile, 2000))
    load()
    if kind == "control":
        sim.set_control((0.5 * sc.sys.Lx, 0.5 * sc.sys.Ly), 5e-3)
    sim.step(8)  # five tiles of 4,096 keys: the tiles behind the held one wait
    gave_up()
    if kind != "batch":
        sim.step_followed(7, ids)
        sim.cells()
    sim.step(5)
    sim.get_state()
    gave_up()
    if kind == "adjoint":
        lam = [torch.ones((n, 2), device="cuda"), torch.ones((n, 2), device="cuda"),
               torch.ones(n, device="cuda")]
        sim.adjoint_forward(12, 6)
        sim.adjoint_backward(*lam)
        gave_up()
    D.check(L.dem_debug_sort_hold(sim.handle, NO_HOLD, 0))
    if kind == "control":
        sim.set_control(None, 0)
    load()
    sim.step(12)
    torch.cuda.synchronize()
    sim.check()
    got = sim.get_state("cpu")
    sim.close()
    a = 0
    for p in parts:
        ref = PortOracle("f32").run(p.sys, p.state(), 12)
        for k in ("pos", "vel", "theta", "omega", "pressure"):
            assert same(got[k].numpy()[a:a + p.n], ref[k]), k
        a += p.n
