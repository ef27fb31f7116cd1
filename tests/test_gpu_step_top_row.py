"""A disk whose radius the box height swallows (Ly - r == Ly) sits in the grid's
first row once the top wall holds it, and meets the disks of the last row across
the wrap: a neighbour that comes near without changing cell is met when it is in
reach, in a single scene and in every specimen of a batch."""
import numpy as np
import pytest

from demso_b200 import scenes
from helpers import gpu_run, same
from oracle.oracle import PortOracle

pytestmark = pytest.mark.gpu


def _scene(seed, speed=10.0):
    """64 x 64 cells of 2.2 mm (4 bands in a batch, 16 alone)."""
    sc = scenes.agitated_gas(n=6, seed=seed, grid=(64, 64), box=0.1408, attraction=20.0,
                             gravity=(0.0, 0.0))
    L = np.float32(0.1408)
    w = 0.1408 / 64
    x0 = (20 + seed) * w
    sc.pos[:] = [[x0 + 0.5 * w, L], [x0 - 0.95 * w, 0.1408 - 1.3e-3], [0.03, 0.05], [0.1, 0.09],
                 [0.02, 0.1], [0.11, 0.02]]
    sc.radius[:] = np.float32(1e-3)
    sc.radius[0] = np.float32(1e-9)
    assert np.float32(L - sc.radius[0]) == L
    sc.vel[:] = 0.0
    sc.vel[1] = [speed, 0.0]  # 20 um a step towards the first disk
    sc.omega[:] = 0.0
    sc.mass[:] = scenes.disk_mass(np.full(6, 1e-3))
    sc.mass[0] = 1e-5
    return sc


def _t(a):
    import torch
    a = np.ascontiguousarray(a)
    return torch.from_numpy(a.view(np.int32).copy() if a.dtype == np.uint32 else a.copy())


@pytest.mark.parametrize("specimens", [0, 1, 3])
def test_a_neighbour_in_the_last_row(specimens):
    import torch
    import demso_b200 as D
    # of three only the second moves: its bands' neighbours in memory are at rest
    parts = [_scene(s, 10.0 if specimens < 3 or s == 1 else 0.0) for s in range(max(1, specimens))]
    steps = 85
    if not specimens:
        got = gpu_run(parts[0].sys, parts[0].state(), steps)
    else:
        st = scenes.concat_specimens(parts)
        sim = D.Batch([(p.sys, p.n) for p in parts])
        sim.set_state(*(_t(st[k]) for k in ("pos", "vel", "theta", "omega", "radius", "mass",
                                            "id")))
        sim.step(steps)
        torch.cuda.synchronize()
        sim.check()
        got = {k: v.numpy() for k, v in sim.get_state("cpu").items() if v is not None}
        sim.close()
    for s, p in enumerate(parts):
        ref = PortOracle("f32").run(p.sys, p.state(), steps)
        first = np.nonzero(ref["id"] == 0)[0][0]
        assert np.any(ref["vel"][first] != 0) == (p.vel[1, 0] != 0)  # it was met
        assert np.all(np.floor(ref["pos"][:, 0] * 64 / 0.1408)[ref["id"] == 1] == 19 + s)
        for k in ("pos", "vel", "theta", "omega", "pressure"):
            assert same(got[k][6 * s:6 * s + 6], ref[k]), (s, k)
