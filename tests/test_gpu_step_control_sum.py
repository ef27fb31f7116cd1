"""The control particle's sums over many block results: bit for bit against
the CPU restatement of the reference."""
import numpy as np
import pytest

from demso_b200 import scenes
from oracle.oracle import PortOracle, orc_control

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [512, 524288, 524289 + 512])
def test_control_sums_over_a_tile_of_blocks(n):
    # 1, 1,024 (one tile of the sum) and 1,026 blocks of 512
    sc = scenes.agitated_gas(n=n, seed=9, vel_std=0.3, jitter=0.05, pitch_factor=1.05)
    L = sc.sys.Lx
    c = dict(pos=(0.5 * L, 0.5 * sc.sys.Ly), vel=(0.0, 0.0), theta=0.0, omega=2.0,
             radius=6e-3, mat=0, drift=(2e-5, -5e-5), wrap_y=(-1.0, 0.1), wrap_x=(2 * L, -0.5))
    import torch
    import demso_b200 as D
    sim = D.Simulation(sc.sys, capacity=n, flags=D.CTX_PRESSURE)
    t = lambda a: torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a)
    sim.set_state(t(sc.pos), t(sc.vel), t(sc.theta), t(sc.omega), t(sc.radius), t(sc.mass),
                  t(sc.id))
    sim.set_control(c["pos"], c["radius"], omega=c["omega"], drift=c["drift"],
                    wrap_y=c["wrap_y"], wrap_x=c["wrap_x"])
    got = []
    for _ in range(2):
        sim.step(1)
        got.append(sim.control()[1])
    sim.close()
    _, reac = PortOracle("f32").run_control(sc.sys, sc.state(), 2, orc_control(c))
    assert np.array_equal(np.array(got, np.float32), reac)
    assert np.any(reac != 0)
