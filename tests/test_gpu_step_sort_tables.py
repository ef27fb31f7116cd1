"""The stage sort around the table sizes that are scanned by a warp and by a block
a row (more than 1,024 tiles of 4,096 pairs; 2,048 tiles a turn of a block), and
where the digits' offsets are made beside them (from 4,096 tiles on)."""
import numpy as np
import pytest

from helpers import dev, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [1, 8, 11, 20])
@pytest.mark.parametrize("n", [1024 * 4096, 1024 * 4096 + 1, 2048 * 4096, 2049 * 4096 + 7,
                               4095 * 4096, 4096 * 4096 + 1])
def test_sort_of_many_tiles(n, bits):
    import torch
    import demso_b200 as D
    rng = np.random.default_rng(bits)
    keys = rng.integers(0, 1 << bits, size=n, dtype=np.uint32)
    k, v = dev(keys), dev(np.arange(n, dtype=np.uint32))
    D.sortParticles(k, v, n, keyBits=bits)
    torch.cuda.synchronize()
    order = np.argsort(keys, kind="stable").astype(np.uint32)
    assert np.array_equal(host(v), order) and np.array_equal(host(k), keys[order])
