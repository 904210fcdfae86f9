"""The launches that a graph reports are the kernels that ran for it: for every
stage, on a graph of a size that takes the one-block forms and one that does not,
against the profiler's list of kernels, and the same whatever failed on another
graph before."""
import ctypes

import numpy as np
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

import rtrex_cuda_b200 as rtr
from rtrex_cuda_b200 import graphgen
from tests.test_gpu_priority_rows import CASES, _hubs

pytestmark = pytest.mark.gpu


def _small():
    return graphgen.rmat(scale=9, edge_factor=6, seed=1)


def _medium():
    return graphgen.chung_lu(n=30000, target_edges=80000, n_comm=170, seed=2)


def _rows_ahead():
    n, u, v = _hubs(CASES["40"], 5)
    a, b = np.meshgrid(np.arange(512), np.arange(1024))
    return n + 1536, np.concatenate([u, n + a.ravel()]), np.concatenate([v, n + 512 + b.ravel()])


GRAPHS = {"small": _small, "medium": _medium, "rows_ahead": _rows_ahead}


def _decompose(e):
    g = rtr.Graph.from_edges(*e)
    g.decompose(0.3)
    g.clusters()
    g.cluster_of()
    return g


def _expand(threshold):
    def f(e):
        g = _decompose(e)
        g.expand(threshold)
        return g
    return f


def _rows(cap):
    def f(e):
        g = rtr.Graph.from_edges(*e)
        g.set_count_mode(2, 16)
        g.set_count_window(cap)
        g.count()
        return g
    return f


def _sets(e):
    g = rtr.Graph.from_edges(*e)
    g.set_count_sets(0)
    g.count()
    return g


def _components(e):
    g = rtr.Graph.from_edges(*e)
    k = ctypes.c_int64()
    assert rtr.lib().rtr_connected_components(g._h, ctypes.byref(k)) == 0
    return g


def _nucleus(e):
    g = rtr.Graph.from_edges(*e)
    g.nucleus()
    return g


def _text(e):
    n, u, v = e
    return rtr.Graph.from_escape_text(b"%d %d\n" % (n, u.size) + b"".join(b"%d %d\n" % p for p in zip(u, v)))


def _batch(e):
    g = rtr.Graph.batch([e, _small(), e])
    g.decompose(0.3)
    g.batch_cluster_counts()
    return g


STAGES = {"decompose": _decompose, "expand": _expand(1), "expand_in_order": _expand(0), "rows": _rows(0), "sets": _sets,
          "components": _components, "nucleus": _nucleus, "text": _text, "batch": _batch}


def _kernels(stage, edges):
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        with stage(edges) as g:
            reported = g.stats()["launches"]
        torch.cuda.synchronize()
    ran = [e.name for e in p.events() if e.device_type == torch.autograd.DeviceType.CUDA]
    return reported, sum("::k_" in x for x in ran), ran


@pytest.mark.parametrize("stage,graph", [(s, g) for s in sorted(STAGES) for g in ("small", "medium")] +
                         [("rows", "rows_ahead"), ("sets", "rows_ahead")])
def test_reported_launches_are_the_kernels_that_ran(stage, graph):
    edges = GRAPHS[graph]()
    _kernels(STAGES[stage], edges)  # the profiler's and the pool's first use
    reported, ran, names = _kernels(STAGES[stage], edges)
    if not names:
        pytest.skip("the profiler lists no device activity here")
    assert ran > 0 and reported == ran, sorted(set(names))


def test_a_failed_call_leaves_nothing_to_the_next_graph():
    edges = _small()
    with _decompose(edges) as g:
        want = g.stats()["launches"]
    with rtr.Graph.from_edges(*_medium()) as bad:
        bad.set_count_mode(2)
        bad.set_device_limits(max_alloc=300000)
        with pytest.raises(rtr.RtrError):
            bad.count()
    with _decompose(edges) as g:
        assert g.stats()["launches"] == want
