"""The pressure of a disk without a radius that touches another without a force
(no stiffness, no approach): 0 / 0, as in the reference, on the bands' and the
stages' dealt contact law."""
import numpy as np
import pytest

from demso_b200 import scenes
from helpers import gpu_run, gpu_stages, same
from oracle.oracle import PortOracle

pytestmark = pytest.mark.gpu


def test_pressure_of_a_disk_without_a_radius():
    sc = scenes.agitated_gas(n=3, seed=1, grid=(16, 16), box=0.04, gravity=(0.0, 0.0))
    sc.pos[:] = [[0.02, 0.02], [0.0205, 0.02], [0.01, 0.01]]
    sc.radius[:] = [0.0, 1e-3, 1e-3]
    sc.mass[:] = 1e-5
    sc.vel[:] = 0.0
    sc.omega[:] = 0.0
    m = sc.sys.materials[0]
    m.normalStiffness = m.frictionCoefficient = 0.0
    ref = PortOracle("f32").run(sc.sys, sc.state(), 6)
    assert np.isnan(ref["pressure"]).sum() == 1
    for chunks in ([6], [1] * 6):
        got = gpu_run(sc.sys, sc.state(), 6, chunks=chunks)
        for k in ("pos", "vel", "omega", "pressure"):
            assert same(got[k], ref[k]), (chunks, k)
    st = gpu_stages(sc.sys, sc.state())
    ref = PortOracle("f32").run(sc.sys, sc.state(), 1)
    assert same(st["int_pressure"], ref["pressure"])


@pytest.mark.parametrize("n", [3, 40])
def test_attraction_beside_a_position_that_is_no_number(n):
    # through the five stages, whose cell ranges hold the disk; 40: groups of eight
    sc = scenes.agitated_gas(n=n, seed=2, grid=(4, 4), box=0.012, gravity=(0.0, 0.0),
                             attraction=20.0)
    sc.radius[0] = 0.0
    sc.pos[1] = [np.nan, np.nan]
    sc.vel[:] = 0.0
    sc.omega[:] = 0.0
    st = gpu_stages(sc.sys, sc.state())
    ref = PortOracle("f32").run(sc.sys, sc.state(), 1)
    assert np.isnan(ref["pressure"]).any()
    assert same(st["int_pressure"], ref["pressure"])
