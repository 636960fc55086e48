"""The step's scan where its sums leave an int (scan.cuh): they stop at a limit beyond every buffer's
capacity instead of wrapping, so that too many pairs are an overflow and no row starts below zero."""
import ctypes

import numpy as np
import pytest

MOST = 0x7F000000
_ip = ctypes.POINTER(ctypes.c_int)


@pytest.fixture(scope="module")
def probe(built):
    from shapes_gb300 import build as B

    return ctypes.CDLL(str(B.PROBE_LIB))


def _p(a):
    return a.ctypes.data_as(_ip)


def _prefix(v):
    return np.minimum(np.concatenate([[0], np.cumsum(v.astype(np.int64))]), MOST)


@pytest.mark.parametrize("seed", range(4))
def test_sums_stop_and_are_associative(probe, seed):
    rng = np.random.default_rng(seed)
    n = int(rng.integers(1, 300))
    v = np.minimum(rng.integers(0, 2 ** rng.integers(1, 32, n), dtype=np.int64), MOST).astype(np.int32)
    out, tree = np.empty(n + 1, np.int32), ctypes.c_int()
    probe.shapes_probe_scan_sum(_p(v), n, _p(out), ctypes.byref(tree))
    want = _prefix(v)
    assert np.array_equal(out, want) and tree.value == want[-1]


def test_limit_is_between_the_capacities_and_the_largest_int():
    """Buffers hold at most 2^30 pairs; a position in a row is below 2^20."""
    assert 2 ** 30 < MOST and MOST + 2 ** 20 < 2 ** 31


@pytest.mark.gpu
@pytest.mark.parametrize("n,most", [(0, 1), (1, 2 ** 20), (8191, 3), (8192, 2 ** 20), (8193, 2 ** 17), (65537, 2 ** 16),
                                    (300_000, 2 ** 13), (300_000, 2 ** 20), (300_000, 7)])
def test_scan(probe, n, most):
    """Prefixes below the limit, that reach it inside a tile, between tiles and within the 32 tiles of a look-back."""
    rng = np.random.default_rng(n)
    v = rng.integers(0, most, n, dtype=np.int64).astype(np.int32)
    out, words = np.empty(n + 1, np.int32), (ctypes.c_ulonglong * 3)()
    cap = 2 ** 30 - 1
    assert probe.shapes_probe_scan(_p(v), n, max(n, 1) + 9000, cap, _p(out), words) == 0
    want = _prefix(v)
    assert np.array_equal(out, want)
    assert list(words) == [want[-1], int(want[-1] > cap), 0]
