"""Rays at the ends of the single-precision range: directions far from unit length and scenes of large
coordinates, in every traversal width."""
import numpy as np
import pytest

from seesharp_gb300 import (DiffuseEmitter, DiffuseMaterial, FrameBuffer, Matrix4x4, Mesh, PerspectiveCamera, RgbColor, Scene, Triangle, _native)

pytestmark = pytest.mark.gpu

WIDTHS = (2, 4, 8)


def _soup(centres, size, rng):
    n = len(centres)
    return _scene((centres[:, None, :] + rng.uniform(-size, size, (n, 3, 3))).astype(np.float32))


def _scene(V):
    sc = Scene()
    m = Mesh(V.reshape(-1, 3), np.arange(3 * len(V), dtype=np.int32))
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


def test_hits_do_not_depend_on_the_length_of_the_direction():
    """A direction scaled by a power of two scales every distance of the ray exactly: the same triangle and
    barycentrics, and the distance divided by the same power.  A third of the rays run along an axis plane
    or an axis (components of either zero)."""
    rng = np.random.default_rng(5)
    sc = _soup(rng.uniform(-20, 20, (4000, 3)), 1.0, rng)
    n = 6000
    org = rng.uniform(-20, 20, (n, 3)).astype(np.float32)
    d = rng.standard_normal((n, 3)).astype(np.float32)
    k = np.arange(n)
    first = rng.integers(0, 3, n)
    zero = np.where(rng.random(n) < 0.5, np.float32(0), np.float32(-0.0))
    d[k[: n // 3], first[: n // 3]] = zero[: n // 3]
    d[k[: n // 6], (first[: n // 6] + 1) % 3] = zero[: n // 6]
    want, blocked = _query(sc, _rays(org, d), 2)
    assert (_ids(want)[:, 0] >= 0).sum() > 1000 and (_ids(want)[: n // 6, 0] >= 0).sum() > 200
    for exponent in (0, -40, -96, -100, 40, 90):
        scale = np.float32(2.0 ** exponent)
        for width in WIDTHS:
            hits, occ = _query(sc, _rays(org, d * scale), width)
            assert np.array_equal(hits[:, 0], want[:, 0] / scale), (exponent, width)
            assert np.array_equal(hits[:, 1:].view(np.uint32), want[:, 1:].view(np.uint32)), (exponent, width)
            assert np.array_equal(occ, blocked), (exponent, width)


@pytest.mark.parametrize("width", WIDTHS)
def test_small_components_beside_ordinary_ones_hit_what_fp64_hits(width):
    """Components so small that the product of their inverse with the origin is large or overflows, beside
    ordinary ones: primitive exact and t to a relative 1e-5 on non-degenerate rays (the repository's
    intersection criterion)."""
    from oracle import pyoracle as O
    from seesharp_gb300 import workloads
    sc = workloads.sphere_field(3, 64, 64, seed=2)
    sc.Prepare()
    rng = np.random.default_rng(12)
    n = 900
    d = rng.standard_normal((n, 3)).astype(np.float32)
    small = np.array([1e-38, -1e-38, 3e-37, -3e-37, 1e-35, -1e-33, 1e-31, -1e-30], np.float32)
    first = rng.integers(0, 3, n)
    for axes in (first, np.where(rng.random(n) < 0.5, (first + 1) % 3, first)):
        d[np.arange(n), axes] = small[rng.integers(0, len(small), n)]
    rays = _rays(rng.uniform(0, 20, (n, 3)).astype(np.float32), d)
    hits, occ = _query(sc, rays, width)
    ref, second = O.OracleScene.from_scene(sc).trace_brute64(rays[:, 0:3].astype(np.float64), rays[:, 4:7].astype(np.float64), with_second=True)
    t, u, v, tri = ref.T
    scale = np.maximum(np.abs(rays[:, 0:3]).max(1), 1.0)
    with np.errstate(invalid="ignore"):
        sure = (tri >= 0) & (np.minimum(np.minimum(u, v), 1 - u - v) >= 1e-4) & (second - t >= 1e-4 * t) & (t >= 0.05 * scale)
    assert sure.sum() >= 100
    first_tri = np.cumsum([0] + [m.NumFaces for m in sc.Meshes])
    ids = _ids(hits)
    assert np.array_equal(first_tri[ids[sure, 1]] + ids[sure, 0], tri[sure].astype(np.int64))
    assert (np.abs(hits[sure, 0] - t[sure]) <= 1e-5 * t[sure]).all()
    assert np.array_equal(occ != 0, ids[:, 0] >= 0)


def test_hits_do_not_depend_on_the_scale_of_the_scene():
    """A scene and ray origins scaled by a power of two (coordinates of up to 2e10) scale every distance
    exactly.  A third of the rays run along an axis plane or an axis."""
    n = 4000
    want = None
    for exponent in (0, 25, 30):
        scale = np.float32(2.0 ** exponent)
        rng = np.random.default_rng(6)
        corners = rng.uniform(-20, 20, (4000, 1, 3)).astype(np.float32) + rng.uniform(-1, 1, (4000, 3, 3)).astype(np.float32)
        sc = _scene(corners * scale)
        org = rng.uniform(-20, 20, (n, 3)).astype(np.float32) * scale
        d = rng.standard_normal((n, 3)).astype(np.float32)
        k, first = np.arange(n), rng.integers(0, 3, n)
        d[k[: n // 3], first[: n // 3]] = 0
        d[k[: n // 6], (first[: n // 6] + 1) % 3] = -0.0
        for width in WIDTHS:
            hits, occ = _query(sc, _rays(org, d), width)
            got = (hits[:, 0] / scale, hits[:, 1:3].view(np.uint32), _ids(hits), occ)
            want = want or got
            assert (_ids(hits)[: n // 6, 0] >= 0).any()
            for a, b in zip(got, want):
                assert np.array_equal(a, b), (exponent, width)
