"""The control particle on steps in bands (calls of several steps): state, last
reaction and the control particle's own motion at the end of every call against
the oracle; several blocks of 512 disks, types with attraction, layouts on every
step, and single steps after longer calls, first in the bands, then packed."""
import numpy as np
import pytest

from demso_b200 import scenes
from helpers import same
from oracle.oracle import PortOracle, orc_control

pytestmark = pytest.mark.gpu

FIELDS = ("pos", "vel", "theta", "omega", "radius", "mass", "id", "type")


def _t(a):
    import torch
    a = np.ascontiguousarray(a)
    return torch.from_numpy(a.view(np.int32).copy() if a.dtype == np.uint32 else a.copy())


# n, materials, attraction, velocity edited in after the state is set, calls
CASES = [(300, 1, 0.0, 0.3, (20, 5, 7)), (4000, 1, 0.0, 0.3, (5, 20, 11)),
         (3000, 3, 15.0, 0.3, (20, 12)), (3000, 1, 0.0, 250.0, (9, 6)),
         (2500, 2, 0.0, 250.0, (8,)), (1500, 1, 0.0, 1.0, (6,) + (1,) * 18)]


@pytest.mark.parametrize("n,n_mat,attraction,vel,calls", CASES)
def test_control_particle_in_bands(n, n_mat, attraction, vel, calls):
    import torch
    import demso_b200 as D
    sc = scenes.agitated_gas(n=n, seed=70 + n_mat, n_mat=n_mat, attraction=attraction, vel_std=0.3)
    L, H = sc.sys.Lx, sc.sys.Ly
    c = dict(pos=(0.5 * L, 0.5 * H), vel=(0.0, 0.0), theta=0.0, omega=2.0, radius=5e-3,
             mat=n_mat - 1, drift=(2e-5, -5e-5), wrap_y=(0.45 * H, 0.55 * H),
             wrap_x=(0.5 * L + 4e-4, 0.5 * L))
    sim = D.Simulation(sc.sys, capacity=n, flags=D.CTX_PRESSURE | D.CTX_ACCEL)
    cur = sc.state()
    sim.set_state(*(_t(cur[k]) for k in FIELDS if cur[k] is not None))
    # through the view: the path was chosen for the slow state
    cur["vel"] = (cur["vel"] * np.float32(vel / 0.3)).astype(np.float32)
    sim.state_view()["vel"].mul_(float(np.float32(vel / 0.3)))
    sim.set_control(c["pos"], c["radius"], material=c["mat"], vel=c["vel"], theta=c["theta"],
                    omega=c["omega"], drift=c["drift"], wrap_y=c["wrap_y"], wrap_x=c["wrap_x"])
    oc, ref, met = orc_control(c), PortOracle("f32"), False
    for k in calls:
        sim.step(k)
        pos, reaction = sim.control()
        got = {x: v.numpy() for x, v in sim.get_state("cpu").items() if v is not None}
        torch.cuda.synchronize()
        cur, reac = ref.run_control(sc.sys, cur, k, oc)
        for x in ("pos", "vel", "theta", "omega", "pressure"):
            assert same(got[x], cur[x]), x
        assert np.array_equal(got["id"].view(np.uint32), cur["id"])
        assert np.array_equal(np.array(reaction, np.float32), reac[-1])
        assert pos == (np.float32(oc.pos[0]), np.float32(oc.pos[1]))
        met = met or bool(np.any(reac))
    assert met
    sim.check()
    sim.close()


@pytest.mark.parametrize("n_mat", [1, 3])
def test_layouts_on_every_step(n_mat):
    # 300 m/s: a quarter of the disks change cell on a step, more than a band's
    # events; edited in, so that the call starts in bands
    import demso_b200 as D
    sc = scenes.agitated_gas(n=9001, seed=7, vel_std=1.0, n_mat=n_mat, pitch_factor=1.15,
                             jitter=0.05)
    sim = D.Simulation(sc.sys, capacity=sc.n)
    st = sc.state()
    sim.set_state(*(_t(st[k]) for k in FIELDS if st[k] is not None))
    st["vel"] = (st["vel"] * np.float32(300.0)).astype(np.float32)
    sim.state_view()["vel"].mul_(300.0)
    before = sim.state_view()["set"]
    sim.step(41)
    assert sim.state_view()["set"] == before  # in bands
    got = sim.get_state("cpu")
    sim.check()
    sim.close()
    ref = PortOracle("f32").run(sc.sys, st, 41)
    for k in ("pos", "vel", "theta", "omega", "pressure"):
        assert same(got[k].numpy(), ref[k]), k
