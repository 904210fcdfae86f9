"""The rows layout's heavy edges walked against a row of bits in shared memory:
shorter rows of lengths around a word of 32 and a step of 128 elements, runs of
words around the least that is cut into pieces (256) and around a piece (8,192),
vertex counts around a table's size and the largest (2^20; more keep the hash
sets), with ids in random order, beside a complete bipartite graph that brings the
heavy edges to the number from which the bits are used (2^18), or falls short of it
by one -- against the oracle bit for bit."""
import numpy as np
import pytest

import oracle
import rtrex_cuda_b200 as rtr
from tests import helpers

pytestmark = pytest.mark.gpu


def _wheel(spokes, length, n, seed):
    """A hub joined to `spokes` vertices, which form a ring lattice: their rows have `length`
    entries (odd), the hub's among them; ids drawn from [0, n) in random order."""
    i = np.arange(spokes)
    us, vs = [np.zeros(spokes, np.int64)], [1 + i]
    for d in range(1, (length - 1) // 2 + 1):
        us.append(1 + i)
        vs.append(1 + (i + d) % spokes)
    ids = np.random.Generator(np.random.PCG64(seed)).permutation(n)[: spokes + 1]
    return ids[np.concatenate(us)], ids[np.concatenate(vs)]


def _filled(n, u, v, n_total=None, heavy=1 << 18):
    """With K(512, .) beside it (no triangle, every edge heavy): `heavy` edges of it."""
    b = (heavy + 511) // 512
    ids = n + np.arange(512 + b) if n_total is None else np.setdiff1d(np.arange(n_total), np.concatenate([u, v]))
    k = np.arange(heavy)
    return (n + 512 + b if n_total is None else n_total, np.concatenate([u, ids[k % 512]]),
            np.concatenate([v, ids[512 + k // 512]]))


def _check(n, u, v, edge):
    c = oracle.build_csr(n, u, v)
    s = oracle.count(c)
    with rtr.Graph.from_edges(n, u, v) as g:
        g.set_tuning(16, 32, edge)
        g.set_count_mode(2)
        for _ in range(2):
            assert g.count() == s.total
            pe, pv, sup, _ = g.weights()
            assert (helpers.bits(pe) == helpers.bits(s.perEdge)).all()
            assert (helpers.bits(pv) == helpers.bits(s.perVertex)).all()
            assert (sup == s.support).all()


@pytest.mark.parametrize("length", [3, 31, 33, 63, 65, 95, 97, 127, 129, 255, 257])
@pytest.mark.parametrize("spokes", [300, 1100])
def test_row_lengths(spokes, length):
    n = spokes + 1
    u, v = _wheel(spokes, min(length, 255) if spokes == 300 else length, n, length)
    _check(*_filled(n, u, v), 200)


@pytest.mark.parametrize("spokes,length", [(255, 31), (256, 31), (257, 31), (4095, 33), (4096, 33), (4097, 33),
                                           (8193, 3), (3000, 97)])
def test_runs_and_pieces(spokes, length):
    u, v = _wheel(spokes, length, spokes + 100, spokes)
    _check(*_filled(spokes + 100, u, v), 200)


@pytest.mark.parametrize("n", [1 << 13, (1 << 13) + 1, 1 << 19, (1 << 19) + 1, 1 << 20, (1 << 20) + 1])
def test_vertex_counts(n):
    parts = [_wheel(1100, 41, n, 7), _wheel(1100, 9, n, 8), _wheel(700, 21, n, 9)]
    key = np.concatenate([np.minimum(u, v) * n + np.maximum(u, v) for u, v in parts])
    key = np.unique(key)
    _check(*_filled(n, key // n, key % n, n), 300)


@pytest.mark.parametrize("more", [-1, 0, 1])
def test_heavy_edge_counts(more):
    n = 3 * 256 + 5000
    a, b = np.meshgrid(np.arange(256), 768 + np.arange(1000))  # all heavy, with triangles among the first
    i = np.arange(256)
    u = np.concatenate([a.ravel(), i[:-1], i[:-2]])
    v = np.concatenate([b.ravel(), i[1:], i[2:]])
    _check(*_filled(n, u, v, heavy=(1 << 18) - u.size + more), 300)
