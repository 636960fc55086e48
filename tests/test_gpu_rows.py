"""Broadphase rows and their offsets at the edges of their rules: rows that keep
their pairs and rows that do not, rows sorted in shared memory and rows too long
for it, both team widths, and scans that end on, before and after a tile."""
import numpy as np
import pytest

from oracle import oracle as O
from shapes_gb300 import scenes
from tests.parity import batch_from_scene, compare_collision

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    import torch

    torch.cuda.set_device(0)


def _crowds(n: int) -> dict:
    """n bodies: a floor, crowds of 8, 9, 10, 256, 258 and 300 boxes that all
    overlap one another (as far as n allows), in mixed index order, and lone boxes."""
    spots = []
    for k, size in enumerate((8, 9, 10, 256, 258, 300)):
        if len(spots) + size < n - 1:
            spots += [(-300.0 + 20.0 * k + 0.001 * j, 5.0 + 0.0007 * j) for j in range(size)]
    lone = n - 1 - len(spots)
    at = spots + [(-400.0 + 2.0 * (j % 400), 20.0 + 2.0 * (j // 400)) for j in range(lone)]
    order = np.random.default_rng(n).permutation(len(at))
    b = scenes.SceneBuilder()
    half = len(order) // 2
    box = scenes.rectangle_vertices(1.0, 1.0)
    for k in order[:half]:
        b.add(box, at[k])
    b.add(scenes.rectangle_vertices(900.0, 10.0), (0.0, 0.0), static=True)
    for k in order[half:]:
        b.add(box, at[k])
    return b.build(dt=1.0 / 60.0, baumgarte=0.01, slop=0.02, accel=(0.0, -9.8), iterations=4, steps=1)


@pytest.mark.parametrize("n", [11, 63, 1000, 8191, 8192, 8193, 38912, 38913])
def test_rows_match_the_oracle(n):
    sc = _crowds(n)
    ow = O.world_from_scene(sc)
    ow.collide()
    for incremental in (True, False):
        b = batch_from_scene(sc)
        b.set_incremental(incremental)
        for _ in range(2):  # lists built, then lists kept
            b.collide()
            compare_collision(b, [ow], f"{n} bodies, incremental {incremental}")
        b.close()


@pytest.mark.parametrize("cols,rows", [(6, 5), (160, 130)])
def test_constants_and_cache_entries(cols, rows):
    """The contact build with its constants stored directly and staged (capacity from 65,536 contacts on), and
    the search for last step's entries where every contact stays, moves and goes: steps equal the oracle's."""
    from tests.parity import assert_bits_equal, config_of

    sc = scenes.single_world_boxes(seed=9, cols=cols, rows=rows)
    sc["config"]["iterations"] = 2
    b, ow = batch_from_scene(sc), O.world_from_scene(sc)
    c = sc["config"]
    for k in range(3):
        b.step(config_of(sc), 2)
        ow.step(c["dt"], c["baumgarte"], c["slop"], c["accel"], c["iterations"], nsteps=2)
        state = b.get_bodies()
        for f in state:
            assert_bits_equal(state[f], ow.bodies()[f], f"step {2 * k + 2} {f}")
        if k == 1:
            assert b.stats()["cache_hits"] > 0
    b.close()
