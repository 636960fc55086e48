"""Body state through set_bodies and get_bodies: every route (a pinned block for
small handles, driver copies for large ones, arrays of mixed kinds) returns the
bits it was given, refuses what is not finite and follows a growing handle."""
import numpy as np
import pytest
import torch

from shapes_gb300 import _lib, scenes
from tests.parity import assert_bits_equal, batch_from_scene

pytestmark = pytest.mark.gpu

BOX = scenes.rectangle_vertices(1.0, 1.0)


@pytest.fixture(scope="module", autouse=True)
def _dev(built):
    torch.cuda.set_device(0)


def _scene(n):
    b = scenes.SceneBuilder()
    for k in range(n):
        b.add(BOX, (2.0 * (k % 128), 2.0 * (k // 128)))
    return b.build(dt=1.0 / 60.0, baumgarte=0.01, slop=0.02, accel=(0.0, -9.8), iterations=2, steps=1)


@pytest.mark.parametrize("n", [1, 2, 257, 16384, 16385])
def test_state_round_trip(n):
    b = batch_from_scene(_scene(n))
    rng = np.random.default_rng(n)
    state = {f: rng.uniform(0.1, 2.0, n) for f in _lib.BODY_FIELDS}
    b.set_bodies(state)
    got = b.get_bodies()
    for f in _lib.BODY_FIELDS:
        assert_bits_equal(got[f], state[f], f)
    for bad in (np.nan, np.inf, -np.inf):
        refused = {f: a.copy() for f, a in state.items()}
        refused["bounce"][n - 1] = bad
        refused["pos_x"] += 1.0
        with pytest.raises(_lib.ShapesError):
            b.set_bodies(refused)
    mixed = dict(state, pos_y=torch.from_numpy(state["pos_y"] + 3.0).pin_memory().numpy())
    b.set_bodies(mixed)
    got = b.get_bodies()
    for f in _lib.BODY_FIELDS:
        assert_bits_equal(got[f], mixed[f], f)
    b.close()


def test_a_growing_handle():
    n = 5
    b = batch_from_scene(_scene(n))
    want = b.get_bodies()
    for k in range(3):
        row = {f: want[f][0] for f in _lib.BODY_FIELDS}
        row["pos_x"] = -10.0 - 3.0 * k
        slot = b.append_body(0, row, BOX)
        assert slot == n + k
        got = b.get_bodies()
        want = {f: np.append(want[f], row[f]) for f in _lib.BODY_FIELDS}
        for f in _lib.BODY_FIELDS:
            assert_bits_equal(got[f], want[f], f)
        want["vel_x"] = want["vel_x"] + 1.0
        b.set_bodies(want)
        assert_bits_equal(b.get_bodies()["vel_x"], want["vel_x"], "vel_x")
    b.close()
