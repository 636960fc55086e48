"""The narrowphase's binary32 filter against the full binary64 search, bit for bit.

shapes_batch_set_narrowphase_lanes(32) searches every axis and makes every comparison in
binary64, so its contacts are what the filtered path has to reproduce: hulls of up to 64
vertices, exactly touching and exactly aligned boxes, nearly parallel edges, and coordinates
from near the origin to where binary32 cannot tell the hulls apart or overflows.
"""
import numpy as np
import pytest

from oracle import oracle as O
from shapes_gb300 import _lib, scenes

pytestmark = pytest.mark.gpu


def _contacts(sc, lanes):
    b = _lib.Batch(sc["world_body_offsets"], sc["bodies"], sc["vert_offsets"], sc["local_xy"], sc.get("shape_kind"))
    b.set_narrowphase_lanes(lanes)
    b.collide()
    out = b.get_contacts()
    b.close()
    return out


def _check(sc, least):
    (k0, v0, _), (k1, v1, _) = _contacts(sc, 1), _contacts(sc, 32)
    assert len(k0) >= least
    assert np.array_equal(k0, k1)
    assert np.array_equal(v0.view(np.uint64), v1.view(np.uint64))
    if "shape_kind" not in sc:
        ow = O.world_from_scene(sc)
        ow.collide()
        ko, vo = ow.contacts()
        assert np.array_equal(k0, ko)
        assert np.array_equal(np.isnan(v0), np.isnan(vo)) and np.array_equal(v0[~np.isnan(v0)], vo[~np.isnan(vo)])


def _polygons(seed, n, counts, offset, extent=6.0):
    rng = np.random.default_rng(seed)
    b = scenes.SceneBuilder()
    for _ in range(n):
        nv = int(rng.choice(counts))
        ang = np.sort(rng.uniform(0.0, 2.0 * np.pi, nv)) if nv < 5 else 2.0 * np.pi * np.arange(nv) / nv
        if nv < 5:
            ang = 2.0 * np.pi * (np.arange(nv) + rng.uniform(-0.2, 0.2, nv)) / nv
        xy = rng.uniform(0.5, 1.2) * np.stack([np.cos(ang), np.sin(ang)], 1)
        b.add(xy, offset + rng.uniform(0.0, extent, 2), rng.uniform(0.0, 6.28))
    return b.build(dt=1.0 / 60.0, baumgarte=0.01, slop=0.02, accel=(0.0, -9.8), iterations=2, steps=1)


@pytest.mark.parametrize("offset", [0.0, 500.0, 1e5, 1e7, 1e9, 1e14])
@pytest.mark.parametrize("counts", [(3, 4, 5, 6, 7, 8), (8, 9, 16, 17), (33, 64)])
def test_polygons(built, counts, offset):
    _check(_polygons(len(counts), 160, counts, offset), 50)


@pytest.mark.parametrize("angle", [0.0, 1e-12, 1e-9, 1e-6, 1e-4])
@pytest.mark.parametrize("overlap", [0.0, 1e-9, 1e-5, 0.02])
@pytest.mark.parametrize("offset", [0.0, 1000.0])
def test_aligned_boxes(built, offset, overlap, angle):
    """A grid of unit boxes whose sides touch or overlap by a hair, turned by less."""
    rng = np.random.default_rng(3)
    b = scenes.SceneBuilder()
    sq = scenes.rectangle_vertices(1.0, 1.0)
    for k in range(144):
        pitch = 1.0 - overlap
        b.add(sq, (offset + (k % 12) * pitch, offset + (k // 12) * pitch), angle * rng.uniform(-1.0, 1.0))
    _check(b.build(dt=1.0 / 60.0, baumgarte=0.01, slop=0.02, accel=(0.0, -9.8), iterations=2, steps=1), 100)


@pytest.mark.parametrize("scale", [1e-30, 1e-12, 1e14, 1e16, 1e30])
def test_scales(built, scale):
    """Hulls and positions scaled together, past both ends of the filter's range."""
    sc = _polygons(9, 120, (3, 4, 6, 8), 0.0)
    sc["local_xy"] = sc["local_xy"] * scale
    for f in ("pos_x", "pos_y"):
        sc["bodies"][f] = sc["bodies"][f] * scale
    _check(sc, 30)
