"""perVertex in the lists layout: vertices whose term counts lie around the
thread / warp split (64) and the fold's step (128), through the gathered terms
and -- when triangles are rare among the slots -- straight from the lists,
against the oracle bit for bit."""
import numpy as np
import pytest

import oracle
import rtrex_cuda_b200 as rtr
from tests import helpers

pytestmark = pytest.mark.gpu


def _fans(counts, plain_edges):
    """Vertex k: counts[k] triangles over disjoint edges (rows of differing degrees: pendant
    vertices on every third edge's ends), and plain_edges triangle-free edges elsewhere."""
    us, vs, n = [], [], 0
    for c in counts:
        hub = n
        a = hub + 1 + 2 * np.arange(c)
        b = a + 1
        us += [np.full(c, hub), np.full(c, hub), a]
        vs += [a, b, b]
        n += 1 + 2 * c
        third = a[::3]
        us.append(third)
        vs.append(n + np.arange(third.size))
        n += third.size
    us.append(n + np.arange(plain_edges))
    vs.append(n + 1 + np.arange(plain_edges))
    n += plain_edges + 1
    return n, np.concatenate(us).astype(np.int64), np.concatenate(vs).astype(np.int64)


@pytest.mark.parametrize("counts", [[1], [31, 32, 33], [63, 64, 65], [95, 96, 97, 127, 128, 129], [255, 256, 257, 1000]])
@pytest.mark.parametrize("plain", [1, 200000])
def test_fans(counts, plain):
    n, u, v = _fans(counts, plain)
    c = oracle.build_csr(n, u, v)
    s = oracle.count(c)
    with rtr.Graph.from_edges(n, u, v) as g:
        for mode in (0, 1):
            g.set_count_mode(mode)
            assert g.count() == s.total == sum(counts)
            pe, pv, sup, _ = g.weights()
            assert (helpers.bits(pv) == helpers.bits(s.perVertex)).all()
            assert (helpers.bits(pe) == helpers.bits(s.perEdge)).all()
