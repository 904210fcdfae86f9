"""The clean's and the extraction's set-up in one block's launches: seeds and
vertices around the 8,192 up to which it is taken (and 1), with many units and
components and with one, against the oracle bit for bit."""
import numpy as np
import pytest

import oracle
import rtrex_cuda_b200 as rtr
from rtrex_cuda_b200 import graphgen
from tests import helpers

pytestmark = pytest.mark.gpu


def _check(n, u, v, eps):
    c = oracle.build_csr(n, u, v)
    s0 = oracle.count(c)
    s1 = oracle.initial_clean(c, s0, eps)
    ref, s2 = oracle.extract(c, s1, eps)
    with rtr.Graph.from_edges(n, u, v) as g:
        for _ in range(2):
            g.count()
            assert g.clean(eps) == s1.total
            pe, pv, sup, _ = g.weights()
            assert (g.status() == s1.status).all()
            assert (helpers.bits(pe) == helpers.bits(s1.perEdge)).all()
            assert (helpers.bits(pv) == helpers.bits(s1.perVertex)).all()
            assert (sup == s1.support).all()
            assert g.extract() == len(ref)
            cl = g.clusters()
            assert (cl.seed == ref.seed).all() and (cl.off == ref.off).all() and (cl.vert == ref.vert).all()
            assert (cl.ne == ref.ne).all() and (cl.cut == ref.cut).all()
            pe, pv, _, _ = g.weights()
            assert (helpers.bits(pe) == helpers.bits(s2.perEdge)).all()
            assert (helpers.bits(pv) == helpers.bits(s2.perVertex)).all()


def _copies(parts):
    us, vs, n = [], [], 0
    for k, u, v, copies in parts:
        base = n + k * np.arange(copies)[:, None]
        us.append((np.asarray(u) + base).ravel())
        vs.append((np.asarray(v) + base).ravel())
        n += k * copies
    return n, np.concatenate(us).astype(np.int64), np.concatenate(vs).astype(np.int64)


TRIANGLE = (3, [0, 0, 1], [1, 2, 2])  # at eps 0.99 all 3 edges are seeds
DIAMOND = (4, [0, 0, 0, 1, 1], [1, 2, 3, 2, 3])  # the 4 outer ones


@pytest.mark.parametrize("triangles,diamonds", [(1, 0), (2730, 0), (1, 2047), (0, 2048), (2731, 0), (2, 2047), (4000, 1)])
def test_seeds(triangles, diamonds):
    _check(*_copies([TRIANGLE + (triangles,), DIAMOND + (diamonds,)]), 0.99)


@pytest.mark.parametrize("n", [1, 2, 8191, 8192, 8193])
def test_vertices(n):
    """Singletons beside one triangle-free path, and beside cliques that are kept."""
    i = np.arange(min(n - 1, 50))
    _check(n, i, i + 1, 0.3)
    if n > 100:
        a, b = np.triu_indices(24, 1)
        _check(n, np.concatenate([a, a + 30]), np.concatenate([b, b + 30]), 0.1)


@pytest.mark.parametrize("m", [300, 8000, 60000])
def test_one_component(m):
    n, u, v = graphgen.rmat(scale=13, edge_factor=10, seed=m)
    keep = np.sort(np.random.Generator(np.random.PCG64(m)).permutation(u.size)[:m])
    for eps in (0.05, 0.4):
        _check(n, u[keep], v[keep], eps)
