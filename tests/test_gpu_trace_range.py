"""Rays at the ends of the single-precision range: directions far from unit length and scenes of large
coordinates, in every traversal width."""
import numpy as np
import pytest

from seesharp_gb300 import (DiffuseEmitter, DiffuseMaterial, FrameBuffer, Matrix4x4, Mesh, PerspectiveCamera, RgbColor, Scene, Triangle, _native)

pytestmark = pytest.mark.gpu

WIDTHS = (2, 4, 8)


def _soup(centres, size, rng):
    n = len(centres)
    V = (centres[:, None, :] + rng.uniform(-size, size, (n, 3, 3))).astype(np.float32)
    sc = Scene()
    m = Mesh(V.reshape(-1, 3), np.arange(3 * n, dtype=np.int32))
    m.Material = DiffuseMaterial()
    sc.Meshes.append(m)
    sc.Emitters.append(DiffuseEmitter(Triangle(m, 0), RgbColor(1, 1, 1)))
    sc.Camera = PerspectiveCamera(Matrix4x4.CreateLookAt([0, 0, 9], [0, 0, 0], [0, 1, 0]), 40)
    sc.FrameBuffer = FrameBuffer(32, 32)
    sc.Prepare()
    return sc


def _query(sc, rays, width):
    ctx = _native.default_context()
    base = _native.get_tuning(ctx)
    _native.set_tuning(ctx, traceBvhWidth=width)
    try:
        return sc.native.trace(rays), sc.native.occluded(rays)
    finally:
        _native.set_tuning(ctx, **base)


def _rays(org, d):
    rays = np.zeros((len(org), 8), np.float32)
    rays[:, 0:3], rays[:, 4:7], rays[:, 7] = org, d, np.inf
    return rays


def _ids(hits):
    return np.ascontiguousarray(hits[:, 3:5]).view(np.int32)


def test_distances_beyond_the_range_are_misses():
    """Every plane of a box overflows to the same infinity on all three axes: coordinates of 1e10 along
    directions of 1e-29.  No triangle has a finite distance, so every ray misses in every width."""
    rng = np.random.default_rng(3)
    sc = _soup(rng.uniform(-4e10, 4e10, (3000, 3)), 5e9, rng)
    org = rng.uniform(-4e10, 4e10, (2000, 3)).astype(np.float32)
    d = (rng.uniform(1, 2, (2000, 3)) * np.where(rng.random((2000, 3)) < 0.5, -1, 1)).astype(np.float32)
    ordinary = _query(sc, _rays(org, d), 4)[0]
    assert (_ids(ordinary)[:, 0] >= 0).sum() > 500
    for width in WIDTHS:
        hits, occ = _query(sc, _rays(org, d * np.float32(1e-29)), width)
        assert (_ids(hits) == -1).all() and not occ.any()
