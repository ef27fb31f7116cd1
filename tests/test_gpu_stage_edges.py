"""The per-stage sort and collide at their edges: tiles and key widths of the
sort against a stable sort on the host; collide on cell ranges that do not
follow one another in memory against the same particles in sorted order."""
import numpy as np
import pytest

from demso_b200 import scenes
from helpers import EMPTY, dev, gpu_stages, host, same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [1, 6, 7, 11, 20, 32])
@pytest.mark.parametrize("n", [1, 4095, 4096, 4097, 33 * 4096 + 5, 300001])
def test_sort_at_tile_edges(n, bits):
    import torch
    import demso_b200 as D
    rng = np.random.default_rng(n + bits)
    keys = rng.integers(0, 1 << bits, size=n, dtype=np.uint64).astype(np.uint32)
    vals = rng.permutation(n).astype(np.uint32)
    k, v = dev(keys), dev(vals)
    D.sortParticles(k, v, n, keyBits=bits)
    torch.cuda.synchronize()
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(host(k), keys[order]) and np.array_equal(host(v), vals[order])


@pytest.mark.parametrize("n_mat,attraction", [(1, 0.0), (3, 0.0), (1, 20.0), (3, 20.0)])
@pytest.mark.parametrize("n,grid", [(1, (4, 4)), (31, (2, 2)), (33, (1, 4)), (700, (8, 8)),
                                    (700, (16, 2))])
def test_collide_on_scattered_cell_ranges(n, grid, n_mat, attraction):
    import torch
    import demso_b200 as D
    sc = scenes.agitated_gas(n=n, seed=n + grid[0], n_mat=n_mat, attraction=attraction, grid=grid)
    st = gpu_stages(sc.sys, sc.state())
    nc = sc.sys.num_cells
    cs, ce = st["cellStart"], st["cellEnd"]
    # the cells in another order, with foreign particles between them
    rng = np.random.default_rng(1)
    cells = rng.permutation(np.nonzero(cs != EMPTY)[0])
    src, s2, e2 = [], np.full(nc, EMPTY, np.uint32), np.zeros(nc, np.uint32)
    for c in cells:
        src += [int(rng.integers(n))] * int(rng.integers(0, 3))
        s2[c] = len(src)
        src += range(int(cs[c]), int(ce[c]))
        e2[c] = len(src)
    src = np.array(src)
    real = np.zeros(src.size, bool)
    for c in cells:
        real[s2[c]:e2[c]] = True
    m = src.size
    ids = st["sorted_id"][src]
    typ = dev(sc.type[ids]) if n_mat > 1 else None
    acc, alpha, pr = torch.empty((m, 2), device="cuda"), torch.empty(m, device="cuda"), \
        torch.empty(m, device="cuda")
    D.collide(sc.sys, dev(st["sorted_pos"][src]), dev(st["sorted_vel"][src]), acc,
              dev(st["sorted_omega"][src]), alpha, typ, dev(st["sorted_radius"][src]),
              dev(st["sorted_mass"][src]), dev(s2), dev(e2), m, nc, pr)
    torch.cuda.synchronize()
    for a, b in ((acc, st["acc"]), (alpha, st["alpha"]), (pr, st["pressure_collide"])):
        assert same(host(a)[real], b[src][real])
