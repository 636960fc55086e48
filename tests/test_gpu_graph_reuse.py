"""A handle that is stepped now alone, now beside others, and queried in between keeps its step graphs:
each way of stepping captures once a write buffer, and the results stay the oracle's."""
import numpy as np
import pytest

from oracle import oracle as O
from shapes_gb300 import _lib, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("worlds,bodies", [(3, 40), (200, 33)])
def test_alternating_calls_capture_once(built, worlds, bodies):
    sc = scenes.batched_mixed(seed=worlds, n_worlds=worlds, n_bodies=bodies)
    c = sc["config"]
    cfg = _lib.make_config(c["dt"], c["baumgarte"], c["slop"], c["accel"], 3)
    other = _lib.make_config(c["dt"], c["baumgarte"], c["slop"], c["accel"], 3, residual=True)
    bs = [_lib.Batch(sc["world_body_offsets"], sc["bodies"], sc["vert_offsets"], sc["local_xy"]) for _ in range(3)]
    bs[0].step(cfg, 60)  # buffers have grown by then
    for b in bs[1:]:
        b.step(cfg, 60)

    def turn():
        _lib.step_many(bs, cfg, 2)
        bs[0].collide()
        bs[0].step(cfg, 2)
        _lib.step_many(bs[:2], cfg, 2)
        bs[0].step(other, 2)

    turn()
    first = [b.graph_captures() for b in bs]
    for _ in range(4):
        turn()
    assert [b.graph_captures() for b in bs] == first
    got = bs[0].get_bodies()
    for b in bs:
        b.close()
    off, vo = sc["world_body_offsets"], sc["vert_offsets"]
    for w in {0, worlds - 1}:
        s, e = off[w], off[w + 1]
        one = scenes.assemble([e - s], {k: v[s:e] for k, v in sc["bodies"].items()}, sc["local_xy"][vo[s]:vo[e]],
                              np.diff(vo)[s:e], **c)
        ow = O.world_from_scene(one)
        ow.step(c["dt"], c["baumgarte"], c["slop"], c["accel"], 3, nsteps=60 + 5 * 8)
        want = ow.bodies()
        for f in _lib.BODY_FIELDS:
            assert np.array_equal(got[f][s:e].view(np.uint64), want[f].view(np.uint64)), (w, f)
