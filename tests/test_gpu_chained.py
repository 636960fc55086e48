"""Kernels that start while the one before them drains: a handle stepped alone (chained launches),
captured in a graph and not, and beside another handle (ordinary launches) gives the same bits."""
import numpy as np
import pytest

from shapes_gb300 import _lib, scenes
from tests.parity import STATE_FIELDS, assert_bits_equal, batch_from_scene, config_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scene", ["boxes", "mixed", "small"])
def test_chained_and_plain_launches_agree(built, scene):
    import torch

    torch.cuda.set_device(0)
    sc = {"boxes": lambda: scenes.single_world_boxes(seed=3, cols=12, rows=10),
          "mixed": lambda: scenes.batched_mixed(seed=4, n_worlds=24, n_bodies=96),
          "small": lambda: scenes.batched_columns(seed=5, n_worlds=40, nmin=1, nmax=9)}[scene]()
    cfg = config_of(sc)
    alone, direct, beside, other = (batch_from_scene(sc) for _ in range(4))
    direct.set_graphs(False)
    for _ in range(3):
        alone.step(cfg, 20)
        direct.step(cfg, 20)
        _lib.step_many([beside, other], cfg, 20)
    want = alone.get_bodies()
    for b, what in ((direct, "without a graph"), (beside, "beside another"), (other, "the other")):
        got = b.get_bodies()
        for f in STATE_FIELDS:
            assert_bits_equal(got[f], want[f], f"{what}: {f}")
        assert np.array_equal(b.get_pairs()[0], alone.get_pairs()[0]), what
    for b in (alone, direct, beside, other):
        b.close()
