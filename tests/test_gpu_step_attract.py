"""Attraction on the context step, where neighbour columns and rows out of
reach are skipped: bit for bit against the CPU restatement of the reference."""
import numpy as np
import pytest

from demso_b200 import scenes
from helpers import gpu_run, same
from oracle.oracle import PortOracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_mat", [1, 3])
@pytest.mark.parametrize("grid", [(2, 4), (2, 2), (4, 4), (4, 16), (16, 8)])
def test_attraction_on_small_and_wrapping_grids(grid, n_mat):
    # 2 cells on an axis: no skipping; 4 or more: skipping; radii from 0.4 to
    # 1.1 mm, so that the two ranges of a pair differ
    sc = scenes.agitated_gas(n=400, seed=31 + grid[0], n_mat=n_mat, attraction=30.0,
                             vel_std=1.0, grid=grid, pitch_factor=1.2, box=0.0481)
    rng = np.random.default_rng(5)
    sc.radius[:] = np.where(rng.random(400) < 0.3, 0.4e-3, sc.radius).astype(np.float32)
    sc.mass[:] = scenes.disk_mass(sc.radius)
    steps = 25
    got = gpu_run(sc.sys, sc.state(), steps)
    ref = PortOracle("f32").run(sc.sys, sc.state(), steps)
    for k in ("pos", "vel", "theta", "omega", "pressure"):
        assert same(got[k], ref[k]), k
