"""Handles stepped from threads of their own share the GPU as those of one shapes_batches_step do: the
launch shapes follow how many are at work, so the threads take about as long, and the results stay the
oracle's."""
import threading
import time

import numpy as np
import pytest

from oracle import oracle as O
from shapes_gb300 import _lib, scenes

pytestmark = pytest.mark.gpu

HANDLES, STEPS = 8, 20


def _threads(f, items):
    ts = [threading.Thread(target=f, args=(x,)) for x in items]
    for t in ts:
        t.start()
    for t in ts:
        t.join()


def _best(f, n=7):
    best = float("inf")
    for _ in range(n):
        t = time.perf_counter()
        f()
        best = min(best, time.perf_counter() - t)
    return best


def test_own_threads_take_as_long_as_one_call(built):
    """1.1 times as long; 1.6 times where each handle takes the GPU for its own."""
    sc = scenes.batched_balls(seed=1, n_worlds=128, n_bodies=128)
    c = sc["config"]
    cfg = _lib.make_config(c["dt"], c["baumgarte"], c["slop"], c["accel"], 8)
    bs = [_lib.Batch(sc["world_body_offsets"], sc["bodies"], sc["vert_offsets"], sc["local_xy"], sc["shape_kind"])
          for _ in range(HANDLES)]
    _lib.step_many(bs, cfg, 90)
    _threads(lambda b: b.step(cfg, STEPS), bs)
    together = _best(lambda: _lib.step_many(bs, cfg, STEPS))
    apart = _best(lambda: _threads(lambda b: b.step(cfg, STEPS), bs))
    for b in bs:
        b.close()
    assert apart < 1.4 * together, (apart, together)


def test_threads_results(built):
    """Counts that come and go while the steps are enqueued."""
    sc = scenes.batched_mixed(seed=5, n_worlds=5, n_bodies=50)
    c = sc["config"]
    cfg = _lib.make_config(c["dt"], c["baumgarte"], c["slop"], c["accel"], 3)
    bs = [_lib.Batch(sc["world_body_offsets"], sc["bodies"], sc["vert_offsets"], sc["local_xy"])
          for _ in range(HANDLES)]

    def work(b):
        for n in (1, 7, 2, 30, 20):
            b.step(cfg, n)
            b.collide()

    _threads(work, bs)
    got = [b.get_bodies() for b in bs]
    for b in bs:
        b.close()
    off, vo = sc["world_body_offsets"], sc["vert_offsets"]
    for w in range(5):
        s, e = off[w], off[w + 1]
        one = scenes.assemble([e - s], {k: v[s:e] for k, v in sc["bodies"].items()}, sc["local_xy"][vo[s]:vo[e]],
                              np.diff(vo)[s:e], **c)
        ow = O.world_from_scene(one)
        ow.step(c["dt"], c["baumgarte"], c["slop"], c["accel"], 3, nsteps=60)
        want = ow.bodies()
        for g in got:
            for f in _lib.BODY_FIELDS:
                assert np.array_equal(g[f][s:e].view(np.uint64), want[f].view(np.uint64)), (w, f)
