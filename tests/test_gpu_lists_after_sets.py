"""The default layout of a large graph whose lists fit after all: hash sets built,
the longest rows counted ahead of the rest, and the triangle lists then kept -- the
path of 2m >= 2^25, reached on small graphs by lowering that line.  Through count,
clean and extraction against the oracle, bit for bit, in a new graph and counted
again, with the degree from which an edge is a heavy one above and below the rows
taken ahead, beside a complete bipartite graph that brings the heavy edges to the
number from which rows are taken ahead."""
import functools

import numpy as np
import pytest

import oracle
import rtrex_cuda_b200 as rtr
from tests import helpers
from tests.test_gpu_priority_rows import CASES, _hubs

pytestmark = pytest.mark.gpu


@functools.lru_cache(maxsize=None)
def _expected(name, eps):
    n, u, v = _hubs(CASES[name], 5)
    a, b = np.meshgrid(np.arange(512), np.arange(1024))
    u, v = np.concatenate([u, n + a.ravel()]), np.concatenate([v, n + 512 + b.ravel()])
    n += 1536
    c = oracle.build_csr(n, u, v)
    s0 = oracle.count(c)
    s1 = oracle.initial_clean(c, s0, eps)
    cl, _ = oracle.extract(c, s1, eps)
    return (n, u, v), s0, s1, cl


@pytest.mark.parametrize("name", ["below", "at", "edges", "40"])
@pytest.mark.parametrize("edge", [1, 1024, 6000])
def test_lists_kept_after_rows_ahead(name, edge):
    eps = 0.01
    (n, u, v), s0, s1, cl = _expected(name, eps)
    with rtr.Graph.from_edges(n, u, v) as g:
        g.set_tuning(16, 32, edge)
        g.set_count_sets(0)
        for again in range(2):
            assert g.count() == s0.total
            assert g.count_mode()[2]  # the lists were kept
            pe, pv, sup, _ = g.weights()
            assert (helpers.bits(pv) == helpers.bits(s0.perVertex)).all()
            assert (helpers.bits(pe) == helpers.bits(s0.perEdge)).all()
            assert (sup == s0.support).all()
            assert g.clean(eps) == s1.total
            assert (g.status() == s1.status).all()
            pe, pv, sup, _ = g.weights()
            assert (helpers.bits(pv) == helpers.bits(s1.perVertex)).all()
            assert (helpers.bits(pe) == helpers.bits(s1.perEdge)).all()
            assert g.extract() == len(cl)
            got = g.clusters()
            assert (got.vert == cl.vert).all() and (got.off == cl.off).all()
