"""A default count whose triangle lists turn out not to fit when they are asked for
takes the rows layout instead, from the same heavy-edge counts, with the same bits;
the mode that insists on lists reports the allocation.  Small graphs of many
triangles, whose lists are far larger than any other buffer, with hash sets and the
longest rows ahead and without."""
import numpy as np
import pytest

import oracle
import rtrex_cuda_b200 as rtr
from tests import helpers
from tests.test_gpu_priority_rows import CASES, _hubs

pytestmark = pytest.mark.gpu


def _clique(k):
    u, v = np.triu_indices(k, 1)
    return k, u.astype(np.int64), v.astype(np.int64)


def _dense_hubs():
    n, u, v = _hubs(CASES["40"], 5)
    a, b = np.meshgrid(np.arange(512), np.arange(1024))
    k, cu, cv = _clique(200)
    return (n + 1536 + k, np.concatenate([u, n + a.ravel(), n + 1536 + cu]),
            np.concatenate([v, n + 512 + b.ravel(), n + 1536 + cv]))


@pytest.mark.parametrize("graph,sets", [("clique", 1 << 25), ("clique", 0), ("hubs", 1 << 25), ("hubs", 0)])
def test_rows_when_the_lists_have_no_room(graph, sets):
    n, u, v = _clique(200) if graph == "clique" else _dense_hubs()
    s = oracle.count(oracle.build_csr(n, u, v))
    limit = 48 * s.total  # the lists take 96 B a triangle, the rows' lists 12
    with rtr.Graph.from_edges(n, u, v) as g:
        g.set_count_sets(sets)
        for mode, room, lists in ((0, limit, False), (0, limit, False), (1, limit, None), (0, 0, True), (0, limit, True),
                                  (2, limit, False)):
            g.set_count_mode(mode)
            g.set_device_limits(max_alloc=room)
            if lists is None:
                with pytest.raises(rtr.RtrError) as ei:
                    g.count()
                assert ei.value.code == 2 and "triangle-list entries" in str(ei.value)
                continue
            assert g.count() == s.total
            assert g.count_mode()[2] == lists
            pe, pv, sup, _ = g.weights()
            assert (helpers.bits(pv) == helpers.bits(s.perVertex)).all()
            assert (helpers.bits(pe) == helpers.bits(s.perEdge)).all()
            assert (sup == s.support).all()
