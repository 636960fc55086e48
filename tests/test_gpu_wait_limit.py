"""The group solve and the coloured large-world solve give their waits up like the ordered solve does: with a
limit of one poll a step returns SHAPES_E_TIMEOUT, every warp returns, the handle steps again with the default
limit, and a fresh handle matches the oracle."""
import numpy as np
import pytest

from oracle import oracle as O
from shapes_gb300 import _lib, scenes

pytestmark = pytest.mark.gpu


def _batch(sc):
    return _lib.Batch(sc["world_body_offsets"], sc["bodies"], sc["vert_offsets"], sc["local_xy"], sc.get("shape_kind"))


def _times_out_and_recovers(b, cfg):
    b.set_wait_limit(1)
    with pytest.raises(_lib.ShapesError) as e:
        b.step(cfg, 3)
    assert e.value.status == _lib.SHAPES_E_TIMEOUT
    b.set_wait_limit(0)
    b.step(cfg, 2)  # no error; the state is no longer the oracle's


@pytest.mark.parametrize("target,warps", [(300, 1), (300, 2), (300, 4), (300, 8), (9000, 4)])
def test_group_solve(built, target, warps):
    """Lists in shared memory, and (9000 bodies a group) in global memory."""
    sc = scenes.batched_mixed(seed=target, n_worlds=30, n_bodies=299)
    c = sc["config"]
    cfg = _lib.make_config(c["dt"], c["baumgarte"], c["slop"], c["accel"], 3)
    b = _batch(sc)
    b.set_launch(target, 0)
    b.set_group_warps(warps)
    b.step(cfg, 60)
    assert b.stats()["contacts"] > 1000
    _times_out_and_recovers(b, cfg)
    b.close()
    b = _batch(sc)
    b.set_launch(target, 0)
    b.set_group_warps(warps)
    b.step(cfg, 70)
    got = b.get_bodies()
    b.close()
    off, vo = sc["world_body_offsets"], sc["vert_offsets"]
    for w in (0, 29):
        s, e = off[w], off[w + 1]
        one = scenes.assemble([e - s], {k: v[s:e] for k, v in sc["bodies"].items()}, sc["local_xy"][vo[s]:vo[e]],
                              np.diff(vo)[s:e], **c)
        ow = O.world_from_scene(one)
        ow.step(c["dt"], c["baumgarte"], c["slop"], c["accel"], 3, nsteps=70)
        want = ow.bodies()
        for f in _lib.BODY_FIELDS:
            assert np.array_equal(got[f][s:e].view(np.uint64), want[f].view(np.uint64)), (w, f)


def test_coloured_large_world(built):
    sc = scenes.container_world(n=6000, width=90.0, steps=1)
    c = sc["config"]
    cfg = _lib.make_config(c["dt"], c["baumgarte"], c["slop"], c["accel"], c["iterations"], coloured=True)
    b = _batch(sc)
    b.step(cfg, 200)
    assert b.stats()["contacts"] > 300
    start, cache = b.get_bodies(), b.get_cache()
    b.step(cfg, 5)
    want = b.get_bodies()
    _times_out_and_recovers(b, cfg)
    b.set_bodies(start)
    b.set_cache(*cache)
    b.step(cfg, 5)
    got = b.get_bodies()
    b.close()
    for f in _lib.BODY_FIELDS:
        assert np.array_equal(got[f].view(np.uint64), want[f].view(np.uint64)), f
