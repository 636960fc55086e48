"""A handle on another device than the calling thread's current one."""
import numpy as np
import pytest

from shapes_gb300 import _lib, scenes

pytestmark = pytest.mark.gpu


def test_get_bodies_from_another_device(built):
    """Small states are read through a kernel; that must not need the caller to switch devices, nor switch them."""
    import torch

    if torch.cuda.device_count() < 2:
        pytest.skip("needs two devices")
    sc = scenes.single_world_boxes(seed=1, cols=3, rows=3)
    with torch.cuda.device(1):
        b = _lib.Batch(sc["world_body_offsets"], sc["bodies"], sc["vert_offsets"], sc["local_xy"])
    with torch.cuda.device(0):
        got = b.get_bodies()
        assert torch.cuda.current_device() == 0
    for f in _lib.BODY_FIELDS:
        assert np.array_equal(got[f], sc["bodies"][f]), f
    b.close()
