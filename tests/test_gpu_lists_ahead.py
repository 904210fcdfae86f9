"""Counting with lists kept: the heavy edges' fill from the count's notes (edges in
and past the noted half, lists of up to and more than 65,535 entries) and the
hubs' folds ahead of the rest (from 16,384 heavy edges on), against the oracle
bit for bit."""
import numpy as np
import pytest

import oracle
import rtrex_cuda_b200 as rtr
from rtrex_cuda_b200 import graphgen
from tests import helpers

pytestmark = pytest.mark.gpu


def _check(n, u, v, edges, gallops=(16,)):
    c = oracle.build_csr(n, u, v)
    s = oracle.count(c)
    with rtr.Graph.from_edges(n, u, v) as g:
        g.set_count_mode(1)
        for edge in edges:
            for gallop in gallops:
                g.set_tuning(gallop, 32, edge)
                assert g.count() == s.total
                pe, pv, sup, _ = g.weights()
                assert (helpers.bits(pe) == helpers.bits(s.perEdge)).all(), (edge, gallop)
                assert (helpers.bits(pv) == helpers.bits(s.perVertex)).all(), (edge, gallop)
                assert (sup == s.support).all(), (edge, gallop)


@pytest.mark.parametrize("m", [16383, 16384, 16385, 60000])
def test_every_edge_heavy(m):
    n, u, v = graphgen.rmat(scale=12, edge_factor=40, seed=5)
    keep = np.sort(np.random.Generator(np.random.PCG64(m)).permutation(u.size)[:m])
    _check(n, u[keep], v[keep], (1, 2, 40, 150, 400, 1024), (1, 16, 10000))


@pytest.mark.parametrize("pages", [65534, 65535, 65536, 70000])
def test_long_lists(pages):
    """A spine of `pages` triangles, and 300 more among the pages' vertices."""
    p = 2 + np.arange(pages)
    r = np.arange(300)
    u = np.concatenate([[0], np.zeros(pages, np.int64), np.ones(pages, np.int64), 2 + 3 * r])
    v = np.concatenate([[1], p, p, 3 + 3 * r])
    _check(2 + pages, u.astype(np.int64), v.astype(np.int64), (1024, 1 << 30))


@pytest.mark.parametrize("m", [(1 << 18) - 1, 1 << 18])
def test_heavy_edges_counted_first(m):
    """Around the number of edges from which the host asks for the heavy ones first: none, some, all."""
    n, u, v = graphgen.rmat(scale=15, edge_factor=12, seed=5)
    keep = np.sort(np.random.Generator(np.random.PCG64(m)).permutation(u.size)[:m])
    assert keep.size == m
    _check(n, u[keep], v[keep], (1, 300, 1024, 1 << 30))
