"""The clean's window replay where every pop pushes: units of few seeds, whose
cascades the first warp of the block pops one by one between windows -- meshes
that unravel from their rim or their holes, random geometric graphs, cliques with
lists around the longest that a warp takes (64 entries) and longer ones -- by the
default rule and with every unit sent to the windows, against the oracle, bit for
bit."""
import functools

import numpy as np
import pytest

import oracle
import rtrex_cuda_b200 as rtr
from tests import helpers

pytestmark = pytest.mark.gpu


def _lattice(w, both=False, drop=0.0):
    """A triangular lattice of w x w vertices (both: both diagonals of each cell), some edges left out."""
    i = np.arange(w * w).reshape(w, w)
    pairs = [(i[:, :-1], i[:, 1:]), (i[:-1], i[1:]), (i[:-1, :-1], i[1:, 1:])]
    if both:
        pairs.append((i[1:, :-1], i[:-1, 1:]))
    u = np.concatenate([a.ravel() for a, _ in pairs])
    v = np.concatenate([b.ravel() for _, b in pairs])
    keep = np.random.default_rng(w).random(u.size) >= drop
    return w * w, u[keep], v[keep]


def _geometric(n, degree, seed):
    """Points of the unit square joined within the radius of that mean degree."""
    p = np.random.default_rng(seed).random((n, 2))
    p = p[np.argsort(p[:, 0])]
    r = np.sqrt(degree / (np.pi * n))
    us, vs = [], []
    last = np.searchsorted(p[:, 0], p[:, 0] + r, side="right")
    for a in range(n):
        b = np.arange(a + 1, last[a])
        b = b[(p[b, 1] - p[a, 1]) ** 2 + (p[b, 0] - p[a, 0]) ** 2 < r * r]
        us.append(np.full(b.size, a))
        vs.append(b)
    return n, np.concatenate(us), np.concatenate(vs)


def _cliques(sizes, eps):
    """Cliques (lists of size - 2).  Pendant vertices, more on some members than on others, bring a tenth of each
    clique's edges below their thresholds; the rest follow them."""
    rng = np.random.default_rng(len(sizes))
    us, vs, pend, n = [], [], [], 0
    for k in sizes:
        a, b = np.triu_indices(k, 1)
        more = rng.integers(0, 30, k)
        while True:  # one pendant vertex at a time
            w = 1.0 / (k - 1 + more)
            if (w.sum() - w[a] - w[b] < eps).mean() > 0.1:
                break
            more[rng.integers(k)] += 1
        us.append(a + n)
        vs.append(b + n)
        pend.append(np.repeat(np.arange(n, n + k), more))
        n += k
    pend = np.concatenate(pend)
    us.append(pend)
    vs.append(n + np.arange(pend.size))
    return n + pend.size, np.concatenate(us), np.concatenate(vs)


GRAPHS = {
    "lattice": (lambda: _lattice(70), 0.3),
    "lattice_deep": (lambda: _lattice(150), 0.3),
    "lattice_holes": (lambda: _lattice(60, drop=0.06), 0.3),
    "king": (lambda: _lattice(50, both=True), 0.4),
    "geometric": (lambda: _geometric(3000, 16, 1), 0.5),
    "geometric_dense": (lambda: _geometric(1500, 60, 2), 0.5),
    "cliques_at": (lambda: _cliques([65, 66, 67, 65, 66, 67], 0.8), 0.8),
    "cliques_long": (lambda: _cliques([12, 80, 30, 100, 12, 70, 66, 150], 0.8), 0.8),
}


@functools.lru_cache(maxsize=2)
def _expected(name):
    n, u, v = GRAPHS[name][0]()
    u, v = u.astype(np.int64), v.astype(np.int64)
    c = oracle.build_csr(n, u, v)
    s0 = oracle.count(c)
    return (n, u, v), c, s0, oracle.initial_clean(c, s0, GRAPHS[name][1])


@pytest.mark.parametrize("split", [None, (1, 1e30)])
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_cascades(name, split):
    (n, u, v), _, s0, s1 = _expected(name)
    with rtr.Graph.from_edges(n, u, v) as g:
        if split is not None:
            g.set_clean_split(*split)
        for again in range(2):
            assert g.count() == s0.total
            assert g.clean(GRAPHS[name][1]) == s1.total
            pe, pv, sup, _ = g.weights()
            assert (g.status() == s1.status).all()
            assert (helpers.bits(pe) == helpers.bits(s1.perEdge)).all()
            assert (helpers.bits(pv) == helpers.bits(s1.perVertex)).all()
            assert (sup == s1.support).all()


def test_stack_overflow_is_reported():
    """A cascade deeper than the ring holds reports it when it may not spill, and is exact when it may."""
    (n, u, v), _, _, s1 = _expected("lattice_deep")
    with rtr.Graph.from_edges(n, u, v) as g:
        g.set_clean_split(1, 1e30)
        g.count()
        g.set_clean_checks(stack_entries=0)
        with pytest.raises(rtr.RtrError) as ei:
            g.clean(0.3)
        assert ei.value.code == 6 and "cascade stack overflowed" in str(ei.value)
        g.set_clean_checks()
        g.count()
        assert g.clean(0.3) == s1.total
        assert (g.status() == s1.status).all()
