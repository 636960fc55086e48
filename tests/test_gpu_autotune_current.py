"""The autotuner times the packing in use and the automatic one among its candidates: it does not leave a
handle slower than it found it, and what it chose can be read back and given to another handle."""
import time

import numpy as np
import pytest

from shapes_gb300 import _lib, scenes

pytestmark = pytest.mark.gpu


def _best(b, cfg, start, cache):
    best = float("inf")
    for _ in range(5):
        b.set_bodies(start)
        b.set_cache(*cache)
        b.step(cfg, 1)
        t = time.perf_counter()
        b.step(cfg, 8)
        best = min(best, time.perf_counter() - t)
    return best


@pytest.mark.parametrize("current", ["automatic", "by bodies"])
def test_no_slower_than_before(built, current):
    """Small worlds of many sweeps: the automatic packing and groups of 190 bodies hold 32 of them, the packings
    by world count at most 4."""
    sc = scenes.batched_columns(seed=3, n_worlds=12000, nmin=4, nmax=8)
    c = sc["config"]
    cfg = _lib.make_config(c["dt"], c["baumgarte"], c["slop"], c["accel"], 64)
    b = _lib.Batch(sc["world_body_offsets"], sc["bodies"], sc["vert_offsets"], sc["local_xy"])
    if current != "automatic":
        b.set_launch(190, 0)
        b.set_group_warps(4)
    b.step(cfg, 60)
    start, cache = b.get_bodies(), b.get_cache()
    before = _best(b, cfg, start, cache)
    b.set_bodies(start)
    b.set_cache(*cache)
    wpg, _, warps = b.autotune(cfg, 4)
    after = _best(b, cfg, start, cache)
    assert after < 1.1 * before, (after, before, wpg, b.group_target(), warps)

    other = _lib.Batch(sc["world_body_offsets"], sc["bodies"], sc["vert_offsets"], sc["local_xy"])
    if wpg:
        other.set_launch_groups(wpg, 0, warps)
    else:
        other.set_launch(b.group_target(), 0)
        other.set_group_warps(warps)
    other.set_world_order(b.world_order())
    other.set_spread_heavy(b.spread_heavy())
    theirs = _best(other, cfg, start, cache)
    got, want = other.get_bodies(), b.get_bodies()
    b.close()
    other.close()
    assert theirs < 1.1 * after, (theirs, after)
    for f in _lib.BODY_FIELDS:
        assert np.array_equal(got[f].view(np.uint64), want[f].view(np.uint64)), f
