"""The nucleus path's units and levels (rtrex_cuda_b200/csrc/nucleus.cu) against
the oracle's restatement, exactly: no triangle at all, one unit, many units of
one and of many levels, cliques that share an edge or a vertex, nested levels
whose clusters take in several children, lists around 32 entries, repeated runs
on one handle."""
import numpy as np
import pytest

import oracle
import rtrex_cuda_b200 as rtr
from rtrex_cuda_b200 import graphgen

pytestmark = pytest.mark.gpu


def _clique(vs):
    a, b = np.triu_indices(len(vs), 1)
    vs = np.asarray(vs)
    return vs[a], vs[b]


def _union(parts, n):
    u, v = graphgen.simplify(n, np.concatenate([p[0] for p in parts]), np.concatenate([p[1] for p in parts]))
    return n, u, v


def _case(name):
    rng = np.random.default_rng(17)
    if name == "path":
        return 50, np.arange(49), np.arange(1, 50)
    if name == "triangle":
        return _union([_clique([0, 1, 2])], 4)
    if name == "many_triangles":
        return _union([_clique([3 * i, 3 * i + 1, 3 * i + 2]) for i in range(70)], 210)
    if name == "clique_sizes":
        sizes, parts, n = list(range(3, 40, 4)), [], 0
        for k in sizes:
            parts.append(_clique(np.arange(k) + n))
            n += k
        return _union(parts, n)
    if name == "share_edge":
        return _union([_clique(range(0, 10)), _clique(list(range(8, 20))), _clique(list(range(18, 25)))], 25)
    if name == "share_vertex":
        return _union([_clique(range(0, 9)), _clique(range(8, 17)), _clique(range(16, 22))], 22)
    if name == "nested":
        # dense cores inside sparser shells inside a random background
        parts = [(rng.integers(0, 300, 2500), rng.integers(0, 300, 2500))]
        for k in range(6):
            core = rng.choice(300, 12, replace=False)
            parts.append(_clique(core))
            parts.append((np.repeat(core[:4], 20), rng.integers(0, 300, 80)))
        return _union(parts, 300)
    if name == "book":
        p = np.arange(34) + 2
        return _union([(np.array([0]), np.array([1])), (np.zeros(34, int), p), (np.ones(34, int), p)], 36)
    if name.startswith("random"):
        n = int(rng.integers(30, 200)) + int(name[6:])
        m = 6 * n
        return _union([(rng.integers(0, n, m), rng.integers(0, n, m))], n)
    if name == "rmat":
        return graphgen.rmat(scale=9, edge_factor=12, seed=3)
    raise KeyError(name)


@pytest.mark.parametrize("name", ["path", "triangle", "many_triangles", "clique_sizes", "share_edge", "share_vertex",
                                  "nested", "book", "random0", "random7", "random90", "rmat"])
def test_against_the_restatement(name):
    n, u, v = _case(name)
    want = oracle.nucleus(oracle.build_csr(n, u, v))
    with rtr.Graph.from_edges(n, u, v) as g:
        for _ in range(2):
            assert g.nucleus() == len(want.id)
            c, nv, ne, par, off, vert = g.nuclei()
            assert (c == want.c).all() and (nv == want.nv).all() and (ne == want.ne).all()
            assert (par == want.parent).all() and (off == want.off).all() and (vert == want.vert).all()
