"""The group solver at the edges of its storage and dealing rules, against the oracle bit for bit.

Groups whose lists fit shared memory with and without the Lagrangians, groups that keep them in
global memory, one to eight solver warps, levels narrower and wider than a round of updates.
"""
import numpy as np
import pytest

from oracle import oracle as O
from shapes_gb300 import _lib, scenes

pytestmark = pytest.mark.gpu


def _run(sc, steps, setup):
    c = sc["config"]
    b = _lib.Batch(sc["world_body_offsets"], sc["bodies"], sc["vert_offsets"], sc["local_xy"], sc.get("shape_kind"))
    setup(b)
    b.step(_lib.make_config(c["dt"], c["baumgarte"], c["slop"], c["accel"], c["iterations"]), steps)
    got, st = b.get_bodies(), b.stats()
    b.close()
    return got, st


def _check(sc, got, steps, worlds):
    c, off, vo = sc["config"], sc["world_body_offsets"], sc["vert_offsets"]
    for w in worlds:
        s, e = off[w], off[w + 1]
        one = scenes.assemble([e - s], {k: v[s:e] for k, v in sc["bodies"].items()}, sc["local_xy"][vo[s]:vo[e]],
                              np.diff(vo)[s:e], **c)
        ow = O.world_from_scene(one)
        ow.step(c["dt"], c["baumgarte"], c["slop"], c["accel"], c["iterations"], nsteps=steps)
        want = ow.bodies()
        for f in _lib.BODY_FIELDS:
            assert np.array_equal(got[f][s:e].view(np.uint64), want[f].view(np.uint64)), (w, f)


@pytest.mark.parametrize("warps", [1, 2, 4, 8])
@pytest.mark.parametrize("cols,rows", [(1, 1), (3, 5), (9, 16), (40, 24)])
def test_one_world(built, cols, rows, warps):
    """Levels of one update to some hundred, up to 961 bodies."""
    sc = scenes.single_world_boxes(seed=cols, cols=cols, rows=rows)
    got, st = _run(sc, 25, lambda b: b.set_group_warps(warps))
    assert st["contacts"] > 0
    _check(sc, got, 25, [0])


@pytest.mark.parametrize("target", [300, 1500, 2200, 9000])
def test_group_sizes(built, target):
    """Groups of 30 worlds of 299 bodies, packed so that everything fits shared memory (300), the lists do
    but not the Lagrangians, or nothing does (9000)."""
    sc = scenes.batched_mixed(seed=target, n_worlds=30, n_bodies=299)
    sc["config"]["iterations"] = 3
    got, st = _run(sc, 90, lambda b: b.set_launch(target, 0))
    assert st["contacts"] > 1000
    _check(sc, got, 90, [0, 7, 29])


def test_one_world_outside_shared_memory(built):
    """A box grid of 4089 bodies, some 8000 contacts: larger than a group's shared memory."""
    sc = scenes.single_world_boxes(seed=1, cols=73, rows=56)
    got, st = _run(sc, 12, lambda b: None)
    assert st["contacts"] > 3000
    _check(sc, got, 12, [0])


@pytest.mark.parametrize("count", [3, 4, 5, 8, 9, 16, 17, 20, 24, 25, 31, 32, 33, 36, 37, 40, 41, 48, 64, 69, 72])
@pytest.mark.parametrize("warps", [4, 8])
def test_levels_of_every_width(built, count, warps):
    """Levels of exactly `count` updates: pairs of boxes that touch nothing else, one contact pair each, dealt
    eight, four and two lanes to an update."""
    b = scenes.SceneBuilder()
    box = scenes.rectangle_vertices(1.0, 1.0)
    for k in range(count):
        b.add(box, (8.0 * k, 0.0), rot=0.0)
        b.add(box, (8.0 * k + 0.02 * (k % 7), 0.995), rot=0.001 * (1 + k % 5))
    sc = b.build(dt=1.0 / 60.0, baumgarte=0.01, slop=0.02, accel=(0.0, -9.8), iterations=6, steps=4)
    got, st = _run(sc, 4, lambda h: h.set_group_warps(warps))
    assert st["contacts"] >= count
    _check(sc, got, 4, [0])


@pytest.mark.parametrize("worlds,bodies", [(200, 60), (480, 71), (480, 72), (700, 140)])
def test_default_packing(built, worlds, bodies):
    """The default packing on both sides of its rule (one group to an SM up to 224 bodies to an SM), and groups
    of which four fit an SM only without their Lagrangians."""
    sc = scenes.batched_mixed(seed=bodies, n_worlds=worlds, n_bodies=bodies)
    sc["config"]["iterations"] = 3
    got, st = _run(sc, 80, lambda b: None)
    assert st["contacts"] > 1000
    _check(sc, got, 80, [0, worlds // 2, worlds - 1])
