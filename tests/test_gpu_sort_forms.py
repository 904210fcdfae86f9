"""The tiled device sort on its own: every form of it -- its own status words per
pass or one region that all passes share, 32-bit and 64-bit words -- at whole
numbers of tiles and a key more or less, on few and on many tiles, with waits that
run out at once (each earlier tile that has not published is counted instead), and
at the key counts where the forms change by themselves; against numpy's stable
sort, exactly."""
import numpy as np
import pytest

import rtrex_cuda_b200 as rtr

pytestmark = pytest.mark.gpu

ONE_REGION, WIDE = (0, -1), (-1, 0)


def _sort(keys, lo, hi, wait=-1, forms=(-1, -1)):
    out = np.zeros_like(keys)
    rc = rtr.lib().rtr_sort_keys(keys.ctypes.data, keys.size, lo, hi, wait, forms[0], forms[1], 0, out.ctypes.data)
    assert rc == 0, rtr.lib().rtr_last_error()
    return out


def _keys(n, lo, hi, seed, skew):
    """Random digits in [lo, hi) -- all alike in most keys when skewed -- over the places below lo,
    which tell equal keys apart."""
    rng = np.random.default_rng(seed)
    top = rng.integers(0, 1 << min(hi - lo, 62), n, dtype=np.uint64)
    if skew:
        top[rng.random(n) < 0.9] = np.uint64((1 << (hi - lo)) - 1)
    low = np.arange(n, dtype=np.uint64) & np.uint64((1 << lo) - 1)
    return (top << np.uint64(lo)) | low


def _expected(keys, lo):
    return keys[np.argsort(keys >> np.uint64(lo), kind="stable")]


@pytest.mark.parametrize("forms", [(-1, -1), ONE_REGION, WIDE, (0, 0)])
@pytest.mark.parametrize("wait", [-1, 0])
@pytest.mark.parametrize("n", [8193, 12287, 12288, 12289, 300001, 4096 * 700])
def test_forms(n, wait, forms):
    for lo, hi in ((0, 20), (24, 47), (32, 64)):
        for skew in (False, True):
            keys = _keys(n, lo, hi, n + lo, skew)
            assert (_sort(keys, lo, hi, wait, forms) == _expected(keys, lo)).all()


@pytest.mark.parametrize("n", [(1 << 24) - 1, 1 << 24, (1 << 24) + 1, (1 << 24) + 2])
def test_where_the_passes_begin_to_share_their_words(n):
    keys = _keys(n, 24, 48, n, False)
    assert (_sort(keys, 24, 48) == _expected(keys, 24)).all()


def test_csr_build_past_the_line():
    """2m = 2^24 and 2^24 + 2 packed pairs through the CSR build: a circulant graph, whose rows are known."""
    for m in (1 << 23, (1 << 23) + 1):
        n, steps = m // 4 + (1 if m % 4 else 0), 4
        src = np.concatenate([np.arange(n)] * steps)[:m].astype(np.int64)
        dst = (src + np.repeat(np.arange(1, steps + 1), n)[:m]) % n
        with rtr.Graph.from_edges(n, src, dst) as g:
            off, nb = g.csr()
        a, b = np.concatenate([src, dst]), np.concatenate([dst, src])
        assert (nb == np.sort(a * np.int64(n) + b) % n).all()
        assert (np.diff(off) == np.bincount(a, minlength=n)).all()
