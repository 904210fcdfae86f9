"""The clean's three kinds of unit in every combination (each kind takes a stream
of its own, the first the graph's), components all large, all small and mixed,
and clusters read back around the size up to which they come as one copy --
against the oracle, bit for bit."""
import numpy as np
import pytest

import oracle
import rtrex_cuda_b200 as rtr
from tests import helpers

pytestmark = pytest.mark.gpu


def _clique(k, pendants):
    a, b = np.triu_indices(k, 1)
    return k + pendants, np.concatenate([a, np.zeros(pendants, np.int64)]), np.concatenate([b, k + np.arange(pendants)])


def _strip(k):
    """A strip of triangles: i joined to i + 1 and i + 2."""
    i = np.arange(k)
    return k, np.concatenate([i[:-1], i[:-2]]), np.concatenate([i[1:], i[2:]])


def _fan(k):
    """One triangle whose corner has k pendant vertices: at most 3 seeds."""
    return 3 + k, np.concatenate([[0, 0, 1], np.zeros(k, np.int64)]), np.concatenate([[1, 2, 2], 3 + np.arange(k)])


def _union(parts):
    us, vs, n = [], [], 0
    for k, u, v in parts:
        us.append(u + n)
        vs.append(v + n)
        n += k
    return n, np.concatenate(us).astype(np.int64), np.concatenate(vs).astype(np.int64)


def _check(n, u, v, eps, clean_split=None, extract_split=None):
    c = oracle.build_csr(n, u, v)
    s0 = oracle.count(c)
    s1 = oracle.initial_clean(c, s0, eps)
    ref, _ = oracle.extract(c, s1, eps)
    with rtr.Graph.from_edges(n, u, v) as g:
        if clean_split:
            g.set_clean_split(*clean_split)
        if extract_split:
            g.set_extract_split(extract_split)
        for _ in range(2):
            g.count()
            assert g.clean(eps) == s1.total
            pe, pv, sup, _ = g.weights()
            assert (g.status() == s1.status).all()
            assert (helpers.bits(pe) == helpers.bits(s1.perEdge)).all()
            assert (helpers.bits(pv) == helpers.bits(s1.perVertex)).all()
            g.extract()
            cl = g.clusters()
            for a, b in zip((cl.nv, cl.ne, cl.cut, cl.off, cl.vert), (ref.nv, ref.ne, ref.cut, ref.off, ref.vert)):
                assert (np.asarray(a) == np.asarray(b)).all()
            own = np.full(n, -1)
            own[cl.vert] = np.repeat(np.arange(len(cl.nv)), cl.nv)
            assert (g.cluster_of() == own).all()


WIDE, NARROW, SMALL = _clique(14, 120), _strip(60), _fan(400)


@pytest.mark.parametrize("kinds", ["w", "n", "s", "wn", "ws", "ns", "wns", "wwnnss"])
@pytest.mark.parametrize("big", [2, 20, 1 << 30])
def test_unit_kinds(kinds, big):
    n, u, v = _union([{"w": WIDE, "n": NARROW, "s": SMALL}[k] for k in kinds])
    _check(n, u, v, 0.9, (5, 1e30), big)


@pytest.mark.parametrize("n", [3, 3275, 3276, 3277, 4096, 5000])
def test_clusters_as_one_copy(n):
    """Singleton clusters: 5n + 1 words against the limit of 16,384."""
    u = np.arange(n - 1)
    _check(n, u, u + 1, 0.3)


@pytest.mark.parametrize("sizes", [[40], [12, 30, 30], [30, 1, 30]])
def test_components_all_large(sizes):
    """Cliques that the clean keeps, a thread block each, with and without a singleton beside them."""
    n, u, v = _union([_clique(k, 0) for k in sizes])
    _check(n, u, v, 0.1, None, 2)
