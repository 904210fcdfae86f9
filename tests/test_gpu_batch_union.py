"""The batch's union on the device: graphs without edges first, last and in
between, single graphs, an endpoint outside its graph (the first such edge is
named), per-graph cluster counts -- each graph against itself alone."""
import ctypes

import numpy as np
import pytest

import rtrex_cuda_b200 as rtr
from rtrex_cuda_b200 import graphgen

pytestmark = pytest.mark.gpu

EMPTY = (3, np.zeros(0, np.int64), np.zeros(0, np.int64))


@pytest.mark.parametrize("pattern", ["g", "eg", "ge", "geeg", "eee", "gggge"])
def test_union_of_graphs_and_empty_graphs(pattern):
    gs = [EMPTY if c == "e" else graphgen.sbm(400 + 37 * i, 80 + i) for i, c in enumerate(pattern)]
    with rtr.Graph.batch(gs) as b:
        off, nb = b.csr()
        b.decompose(0.3)
        counts = b.batch_cluster_counts()
        base = 0
        for (n, u, v), k in zip(gs, counts):
            with rtr.Graph.from_edges(n, u, v) as g:
                o, x = g.csr()
                assert (off[base:base + n + 1] - off[base] == o).all()
                assert (nb[off[base]:off[base + n]] - base == x).all()
                assert g.decompose(0.3) == k
            base += n


@pytest.mark.parametrize("graph,edge,value", [(0, 0, -1), (0, 11, 1 << 40), (2, 0, 10), (2, 5, 10), (3, 19, 30)])
def test_first_bad_endpoint_is_named(graph, edge, value):
    n = np.array([20, 5, 10, 30], np.int64)
    m = np.array([12, 0, 6, 20], np.int64)
    eoff = np.concatenate([[0], np.cumsum(m)])
    src = np.concatenate([np.arange(k) % (x - 1) for k, x in zip(m, n)]).astype(np.int64)
    dst = src + 1
    src[eoff[graph] + edge] = value
    src[-1] = -7 if (graph, edge) != (3, 19) else value  # a later one is not the one reported
    h = ctypes.c_void_p()
    rc = rtr.lib().rtr_batch_create(src.ctypes.data, dst.ctypes.data, eoff.ctypes.data, n.ctypes.data, 4, 0, 1,
                                    ctypes.byref(h))
    assert rc == 3 and not h.value  # RTR_ERR_INPUT
    assert rtr.lib().rtr_last_error().decode() == (
        f"rtr_batch_create: graph {graph} edge {edge} has an endpoint outside [0, {n[graph]})")
