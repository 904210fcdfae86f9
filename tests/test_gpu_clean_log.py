"""The clean without room for the window replay's log: units that would take the
windows replay one warp each, with the same bits, and nothing of the log is held.
Graphs with long and with short lists, alone and beside small units, under the
default rule and with every unit sent to the windows, against the oracle."""
import ctypes

import numpy as np
import pytest

import oracle
import rtrex_cuda_b200 as rtr
from rtrex_cuda_b200 import graphgen
from tests import helpers

pytestmark = pytest.mark.gpu


def _side_by_side(*graphs):
    n = 0
    us, vs = [], []
    for k, u, v in graphs:
        us.append(u + n)
        vs.append(v + n)
        n += k
    return n, np.concatenate(us), np.concatenate(vs)


def _graph(name):
    wide = graphgen.rmat(scale=10, edge_factor=12, seed=3)
    narrow = graphgen.chung_lu(n=4000, target_edges=11000, n_comm=24, seed=4)
    if name == "wide":
        return wide
    if name == "narrow":
        return narrow
    return _side_by_side(wide, narrow, graphgen.sbm(900, 5))


def _peak(g):
    held, peak = ctypes.c_int64(), ctypes.c_int64()
    assert rtr.lib().rtr_get_memory(g._h, ctypes.byref(held), ctypes.byref(peak)) == 0
    return peak.value


@pytest.mark.parametrize("name", ["wide", "narrow", "mixed"])
@pytest.mark.parametrize("split", [None, (1, 1e30)])
def test_units_replay_without_the_log(name, split):
    eps = 0.3
    n, u, v = _graph(name)
    c = oracle.build_csr(n, u, v)
    s0 = oracle.count(c)
    s1 = oracle.initial_clean(c, s0, eps)
    assert s1.total < s0.total
    peaks = []
    for limit in (-1, 0, 40 * s0.total, 1 << 40):
        with rtr.Graph.from_edges(n, u, v) as g:
            if split is not None:
                g.set_clean_split(*split)
            g.set_clean_log(limit)
            for again in range(2):
                g.count()
                assert g.clean(eps) == s1.total
                pe, pv, sup, _ = g.weights()
                assert (g.status() == s1.status).all()
                assert (helpers.bits(pe) == helpers.bits(s1.perEdge)).all()
                assert (helpers.bits(pv) == helpers.bits(s1.perVertex)).all()
                assert (sup == s1.support).all()
            peaks.append(_peak(g))
    full, none, less, most = peaks
    assert none == less < full == most  # the log is taken whole or not at all


def test_setting_the_reported_split_changes_nothing():
    """rtr_set_clean_split of what rtr_get_clean_split reports leaves the library's own rule in force."""
    n, u, v = _graph("wide")
    seen = []
    for split in (None, "reported", (2048, 8.5), "back"):
        with rtr.Graph.from_edges(n, u, v) as g:
            if split == "back":
                g.set_clean_split(1, 1e30)
                g.set_clean_split(2048, 8.0)
            elif split:
                g.set_clean_split(*(g.clean_split() if split == "reported" else split))
            g.count()
            g.clean(0.3)
            seen.append((g.clean_split(), _peak(g)))
    assert seen[0] == seen[1] == seen[3]
    assert seen[2][1] < seen[0][1]  # that unit's lists are longer, it replays one warp
