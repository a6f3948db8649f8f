"""The GPU BVH build around its switch points: the clustering rounds that one block finishes (at most
4096 clusters), sizes just above it, and the levels of the wide trees.  The closest hits of every
traversal width over the clustered tree equal, bit for bit, those over the radix tree, which shares
neither the clustering nor its leaf order (the hit of a ray does not depend on the tree)."""
import numpy as np
import pytest

from seesharp_gb300 import (DiffuseEmitter, DiffuseMaterial, FrameBuffer, Matrix4x4, Mesh, PerspectiveCamera, RgbColor, Scene, Triangle, _native)

pytestmark = pytest.mark.gpu


def _soup(n, coincident):
    rng = np.random.default_rng(n)
    V = (rng.uniform(-3, 3, (n, 1, 3)) + rng.uniform(-0.3, 0.3, (n, 3, 3))).astype(np.float32)
    if coincident:
        V[:] = V[0]
    sc = Scene()
    m = Mesh(V.reshape(-1, 3), np.arange(3 * n, dtype=np.int32))
    m.Material = DiffuseMaterial()
    sc.Meshes.append(m)
    sc.Emitters.append(DiffuseEmitter(Triangle(m, 0), RgbColor(1, 1, 1)))
    sc.Camera = PerspectiveCamera(Matrix4x4.CreateLookAt([0, 0, 9], [0, 0, 0], [0, 1, 0]), 40)
    sc.FrameBuffer = FrameBuffer(32, 32)
    return sc


@pytest.mark.parametrize("n,coincident", [(1, False), (2, False), (3, False), (4, False), (33, False), (1024, False), (4095, False), (4096, False),
                                          (4097, False), (20000, False), (70001, False), (9, True), (5000, True)])
def test_clustered_tree_hits_equal_radix_tree_hits(n, coincident, monkeypatch):
    rng = np.random.default_rng(7)
    rays = np.zeros((3000, 8), np.float32)
    rays[:, 0:3] = rng.uniform(-6, 6, (3000, 3))
    rays[:, 4:7] = rng.uniform(-3, 3, (3000, 3)) - rays[:, 0:3]
    rays[:, 7] = np.inf
    sc = _soup(n, coincident)
    ctx = _native.default_context()
    base = _native.get_tuning(ctx)
    got = []
    try:
        sc.Prepare()
        for width in (2, 4, 8):
            _native.set_tuning(ctx, traceBvhWidth=width)
            got.append(sc.native.trace(rays).view(np.uint32))
    finally:
        _native.set_tuning(ctx, **base)
    monkeypatch.setenv("SST_BVH", "lbvh")
    sc.Prepare()
    want = sc.native.trace(rays).view(np.uint32)
    if n > 2:
        assert (want[:, 4].view(np.int32) >= 0).any()
    for g in got:
        assert np.array_equal(g, want)
