"""The device sort and scan at the edges of their forms -- one block for up to
8,192 keys (16,384 scanned elements), tiles of 4,096 keys with look-back above
-- through the CSR build, which sorts the 2m packed pairs and scans flags over
them: offsets and neighbours against numpy, exactly."""
import numpy as np
import pytest

import rtrex_cuda_b200 as rtr

pytestmark = pytest.mark.gpu


def _graph(m, n, seed):
    rng = np.random.default_rng(seed)
    key = np.zeros(0, np.int64)
    while key.size < m:
        u, v = rng.integers(0, n, 2 * m), rng.integers(0, n, 2 * m)
        k = u != v
        lo, hi = np.minimum(u, v)[k], np.maximum(u, v)[k]
        key = np.unique(np.concatenate([key, lo * n + hi]))
    key = rng.permutation(key)[:m]
    return key // n, key % n


# 2m: one warp, one round and several of the single block, its last size, the
# first tiled sizes, a whole number of tiles and one key more or less, many tiles
@pytest.mark.parametrize("m", [1, 15, 16, 17, 511, 512, 513, 4095, 4096, 4097, 6143, 6144, 6145, 8192, 8193, 40000,
                               524288, 1000003])
@pytest.mark.parametrize("n", [2000, 70000, 20000000])
def test_csr_build(m, n):
    if n == 2000 and m > 500000:
        n = 3000  # room for the edges
    u, v = _graph(m, n, m + n)
    with rtr.Graph.from_edges(n, u, v) as g:
        off, nb = g.csr()
    src, dst = np.concatenate([u, v]), np.concatenate([v, u])
    order = np.lexsort((dst, src))
    assert (nb == dst[order]).all()
    want = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(src, minlength=n), out=want[1:])
    assert (off == want).all()


@pytest.mark.parametrize("m", [100, 4096, 5000, 300001])
def test_repeats_are_dropped(m):
    """The flag scan that drops repeats, with every edge listed twice, reversed the second time."""
    u, v = _graph(m, 50000, m)
    with rtr.Graph.from_edges(50000, np.concatenate([u, v]), np.concatenate([v, u]), simplify=True) as g:
        assert g.m == m
        off, nb = g.csr()
    with rtr.Graph.from_edges(50000, u, v) as g:
        o2, n2 = g.csr()
    assert (off == o2).all() and (nb == n2).all()
