"""Argument checks of the entry points that bound memory and paths (no device needed)."""
import rtrex_cuda_b200 as rtr


def test_null_graphs_are_refused():
    L = rtr.lib()
    assert L.rtr_set_count_sets(None, 0) == 1
    assert L.rtr_set_clean_log(None, -1) == 1
    assert L.rtr_set_device_limits(None, 0, 0) == 1
    assert L.rtr_sort_keys(None, 5, 0, 8, -1, -1, -1, 0, None) == 1
