"""The dependency levels that the group solver finds while it solves, against a walk over all updates of the
step in order (tests/test_level_schedule.py's walk_levels), on the contacts and cache hits of that step."""
import numpy as np
import pytest

from shapes_gb300 import _lib, scenes
from tests.test_level_schedule import walk_levels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("target,warps", [(300, 1), (300, 2), (300, 4), (300, 8), (1500, 4), (9000, 1), (9000, 8)])
@pytest.mark.parametrize("iterations,warm", [(3, True), (2, False), (0, True)])
def test_levels_are_the_walks(built, target, warps, iterations, warm):
    """Groups of one world to 30 of 299 bodies: lists in shared and, of 9000 bodies, in global memory."""
    sc = scenes.batched_mixed(seed=7, n_worlds=30, n_bodies=299)
    c = sc["config"]
    settle = _lib.make_config(c["dt"], c["baumgarte"], c["slop"], c["accel"], 3)
    cfg = _lib.make_config(c["dt"], c["baumgarte"], c["slop"], c["accel"], iterations, warm_start=warm)
    b = _lib.Batch(sc["world_body_offsets"], sc["bodies"], sc["vert_offsets"], sc["local_xy"])
    b.set_launch(target, 0)
    b.set_group_warps(warps)
    b.step(settle, 90)
    cached, _, cached_n = b.get_cache()
    b.step(cfg, 1)
    keys, _, n = b.get_contacts()
    levels = b.world_levels()
    b.close()
    assert n.sum() > 1000 and (cached_n > 0).all()
    moves = (sc["bodies"]["inv_mass_lin"] != 0.0) | (sc["bodies"]["inv_mass_rot"] != 0.0)
    c0, k0 = np.cumsum(n) - n, np.cumsum(cached_n) - cached_n
    for w in range(30):
        had = {tuple(k) for k in cached[k0[w]:k0[w] + cached_n[w]].tolist()}
        off = sc["world_body_offsets"][w]
        contacts = [(i, j, warm and (i, j, fa, fb) in had, bool(moves[off + i]), bool(moves[off + j]))
                    for i, j, fa, fb, _ in keys[c0[w]:c0[w] + n[w]].tolist()]
        assert levels[w] == max(walk_levels(contacts, iterations, warm).values(), default=0), w
