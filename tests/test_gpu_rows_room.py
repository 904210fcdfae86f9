"""The rows ahead take no room that another row needs: on a device of any size that
holds a rows-layout count without them (a set window keeps them out), the count
that may take them ahead succeeds too, with the same bits.  Sizes from too small to
ample, as the graph is told."""
import ctypes

import numpy as np
import pytest

import rtrex_cuda_b200 as rtr
from tests import helpers
from tests.test_gpu_priority_rows import CASES, _hubs

pytestmark = pytest.mark.gpu


def _memory(g):
    held, peak = ctypes.c_int64(), ctypes.c_int64()
    assert rtr.lib().rtr_get_memory(g._h, ctypes.byref(held), ctypes.byref(peak)) == 0
    return held.value, peak.value


def _count(edges, device, window):
    """(perVertex, windows) of a new graph's count, or None where it has no room."""
    with rtr.Graph.from_edges(*edges) as g:
        g.set_count_mode(2)
        g.set_count_window(window)
        g.set_device_limits(graph_bytes=device)
        try:
            g.count()
        except rtr.RtrError as e:
            assert e.code in (2, 4)
            return None
        return g.weights()[1], g.count_windows()[0]


def _edges():
    n, u, v = _hubs(CASES["40"], 5)
    a, b = np.meshgrid(np.arange(512), np.arange(1024))
    return n + 1536, np.concatenate([u, n + a.ravel()]), np.concatenate([v, n + 512 + b.ravel()])


def test_what_fits_without_rows_ahead_fits_with_them():
    edges = _edges()
    with rtr.Graph.from_edges(*edges) as g:
        built, _ = _memory(g)
        g.set_count_mode(2)
        total = g.count()
        want = g.weights()[1]
        held, peak = _memory(g)
    fitted = []
    for device in np.linspace(built, held + peak, 40).astype(np.int64) + (1 << 30):
        alone = _count(edges, int(device), 6 * total)
        ahead = _count(edges, int(device), 0)
        if alone is not None:
            assert ahead is not None, device
            assert (helpers.bits(alone[0]) == helpers.bits(want)).all()
        if ahead is not None:
            assert (helpers.bits(ahead[0]) == helpers.bits(want)).all()
        fitted.append(alone is not None)
    assert not fitted[0] and fitted[-1]  # the sizes span the line


def test_held_buffers_do_for_later_counts():
    """A graph that was counted with rows ahead is counted again when nothing more is available."""
    with rtr.Graph.from_edges(*_edges()) as g:
        g.set_count_mode(2)
        g.count()
        want = g.weights()[1]
        held, _ = _memory(g)
        for device in (0, 1, 1, 0):
            g.set_device_limits(graph_bytes=device)
            g.count()
            assert (helpers.bits(g.weights()[1]) == helpers.bits(want)).all()
            assert _memory(g)[0] == held
