"""The clean's window replay at its edges: list lengths around the 16 threads of
a narrow window item and the 256 of a packed window, more items than a window
holds, edges shared by many items of one window, items whose edges meet in one
slot of the table, and units on both sides of the default rule's 512 seeds --
against the oracle, bit for bit."""
import numpy as np
import pytest

import oracle
import rtrex_cuda_b200 as rtr
from rtrex_cuda_b200 import graphgen
from tests import helpers

pytestmark = pytest.mark.gpu

WINDOW = (1, 1e30)  # every unit takes the window replay


def _check(n, u, v, eps, split=WINDOW):
    c = oracle.build_csr(n, u, v)
    s1 = oracle.initial_clean(c, oracle.count(c), eps)
    with rtr.Graph.from_edges(n, u, v) as g:
        if split is not None:
            g.set_clean_split(*split)
        g.count()
        assert g.clean(eps) == s1.total
        pe, pv, sup, _ = g.weights()
        assert (g.status() == s1.status).all()
        assert (helpers.bits(pe) == helpers.bits(s1.perEdge)).all()
        assert (helpers.bits(pv) == helpers.bits(s1.perVertex)).all()
        assert (sup == s1.support).all()
    return s1


def _cliques(sizes, tails):
    """Cliques with pendant vertices on one member (so that its edges fall below their thresholds first)."""
    us, vs, n = [], [], 0
    for k, t in zip(sizes, tails):
        a, b = np.triu_indices(k, 1)
        us += [a + n, np.full(t, n)]
        vs += [b + n, np.arange(t) + n + k]
        n += k + t
    return n, np.concatenate(us), np.concatenate(vs)


@pytest.mark.parametrize("k", [3, 17, 18, 19, 33, 34])
@pytest.mark.parametrize("eps", [0.3, 0.9])
def test_clique_lists_around_the_item_width(k, eps):
    """A clique of k vertices has lists of k - 2 entries."""
    n, u, v = _cliques([k] * 5, [0, 3, 40, 200, 7])
    _check(n, u, v, eps)


@pytest.mark.parametrize("pages", [15, 16, 17, 255, 256, 257, 600])
def test_book_lists_around_the_window(pages):
    """Books: one edge in `pages` triangles, each page edge in one; three books share a spine vertex."""
    us, vs, n = [], [], 1
    for b in range(3):
        s = n
        p = np.arange(pages) + n + 1
        us += [[0], np.zeros(pages, np.int64), np.full(pages, s)]
        vs += [[s], p, p]
        n += 1 + pages
    _check(n, np.concatenate(us), np.concatenate(vs), 0.3)


@pytest.mark.parametrize("hubs,leaves", [(1, 40), (2, 300), (3, 1200)])
def test_many_items_share_cells(hubs, leaves):
    """Vertices joined to every hub and in a ring: consecutive items subtract from the same hub edges."""
    us, vs = [], []
    leaf = np.arange(leaves) + hubs
    for h in range(hubs):
        us.append(np.full(leaves, h))
        vs.append(leaf)
    us.append(leaf)
    vs.append((leaf - hubs + 1) % leaves + hubs)
    n = hubs + leaves
    su, sv = graphgen.simplify(n, np.concatenate(us), np.concatenate(vs))
    for eps in (0.3, 0.6):
        _check(n, su, sv, eps)


@pytest.mark.parametrize("m,eps", [(900, 0.3), (2600, 0.3), (9000, 0.1)])
def test_dense_rows_meet_in_table_slots(m, eps):
    """R-MAT: long packed lists whose edges collide in the table's slots."""
    n, u, v = graphgen.rmat(scale=8 if m < 5000 else 10, edge_factor=max(4, m // 256), seed=m)
    _check(n, u, v, eps)


@pytest.mark.parametrize("m", [3000, 9001])
def test_default_rule(m):
    """Chung-Lu graphs whose giant units lie on either side of the default rule."""
    n, u, v = graphgen.chung_lu(n=m * 335 // 926, target_edges=m, n_comm=max(1, m // 463), seed=5)
    _check(n, u, v, 0.3, None)
