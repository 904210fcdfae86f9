"""The rows layout's longest rows, counted and folded ahead of the rest: hubs of
2,047 to 2,049 neighbours (the least such row has 2,048) and more than 32 of them
(the most taken), with the degree from which an edge is a heavy one above and
below; counted again in the same graph, in windows, and with lists, beside a
complete bipartite graph that brings the heavy edges to the number from which rows
are taken ahead (2^19), against the oracle bit for bit."""
import numpy as np
import pytest

import oracle
import rtrex_cuda_b200 as rtr
from tests import helpers

pytestmark = pytest.mark.gpu


def _hubs(degrees, seed):
    """Hubs 0..h-1 of exactly the given degrees over a common pool of spokes (neighbours drawn
    without repeats), every pair of hubs joined, and a sparse random graph over the spokes."""
    rng = np.random.Generator(np.random.PCG64(seed))
    h = len(degrees)
    pool = max(degrees) + 700
    us, vs = list(np.triu_indices(h, 1)[:1]), list(np.triu_indices(h, 1)[1:])
    for i, d in enumerate(degrees):
        w = h + rng.choice(pool, d - (h - 1), replace=False)
        us.append(np.full(w.size, i))
        vs.append(w)
    a = rng.integers(0, pool, 4 * pool)
    b = rng.integers(0, pool, 4 * pool)
    key = np.unique(np.minimum(a, b)[a != b] * np.int64(pool) + np.maximum(a, b)[a != b])
    us.append(h + key // pool)
    vs.append(h + key % pool)
    return h + pool, np.concatenate(us).astype(np.int64), np.concatenate(vs).astype(np.int64)


CASES = {
    "below": [2047],
    "at": [2048],
    "edges": [2047, 2048, 2049, 4000],
    "32": [2048 + i for i in range(32)],
    "40": [2100] * 20 + [2048 + 17 * i for i in range(20)],
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("edge", [1, 1024, 2049, 6000])
def test_hubs(name, edge):
    n, u, v = _hubs(CASES[name], 5)
    a, b = np.meshgrid(np.arange(512), np.arange(1024))
    u, v = np.concatenate([u, n + a.ravel()]), np.concatenate([v, n + 512 + b.ravel()])
    n += 1536
    c = oracle.build_csr(n, u, v)
    assert sorted(np.diff(c.offsets)[: len(CASES[name])]) == sorted(CASES[name])
    s = oracle.count(c)
    with rtr.Graph.from_edges(n, u, v) as g:
        g.set_tuning(16, 32, edge)
        for mode, hub, cap in ((2, 1024, 0), (2, 1024, 0), (2, 16, 0), (2, 1024, 2 * s.total), (1, 1024, 0), (2, 1024, 0)):
            g.set_count_mode(mode, hub)
            g.set_count_window(cap)
            assert g.count() == s.total
            pe, pv, sup, _ = g.weights()
            assert (helpers.bits(pv) == helpers.bits(s.perVertex)).all()
            assert (helpers.bits(pe) == helpers.bits(s.perEdge)).all()
            assert (sup == s.support).all()
            if mode == 2:
                windows, entries = g.count_windows()
                assert entries == 3 * s.total and (windows > 1) == (cap > 0)
