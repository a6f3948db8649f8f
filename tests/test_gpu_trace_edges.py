"""Rays that no triangle can meet (an origin that is not finite, a NaN in the direction, a direction of
length zero or with infinite components) end as misses in every traversal width, beside ordinary rays whose hits they do not change.

The CPU part evaluates the watertight edge functions (Woop, Benthin, Wald 2013) in numpy's single
precision for such rays: the distance is never inside any interval, which is what the early end states.
"""
import numpy as np
import pytest

from seesharp_gb300 import _native, workloads

NAN, INF = np.float32(np.nan), np.float32(np.inf)


def _lost_rays():
    out = []
    for k in range(3):
        for bad in (NAN, INF, -INF):
            o, d = np.array([0.1, 0.2, 0.3], np.float32), np.array([0.3, -0.5, 0.8], np.float32)
            o[k] = bad
            out.append((o, d))
        d = np.array([0.3, -0.5, 0.8], np.float32)
        d[k] = NAN
        out.append((np.array([0.1, 0.2, 0.3], np.float32), d))
    out.append((np.zeros(3, np.float32), np.zeros(3, np.float32)))
    for d in ([INF, 0.3, 0.2], [0.1, -INF, 0.2], [INF, INF, 0.2], [-INF, 0.1, INF], [INF, -INF, INF]):
        out.append((np.array([0.1, 0.2, 0.3], np.float32), np.array(d, np.float32)))
    out.append((np.full(3, NAN), np.full(3, NAN)))
    out.append((np.full(3, INF), np.array([0, 0, 1], np.float32)))
    return out


def _distance(o, d, tri):
    """The distance of the watertight test, in single precision, or NaN where it rejects on the edges."""
    f = np.float32
    a = np.abs(d)
    kz = (0 if a[0] > a[2] else 2) if a[0] > a[1] else (1 if a[1] > a[2] else 2)
    kx = 0 if kz == 2 else kz + 1
    ky = 0 if kx == 2 else kx + 1
    if d[kz] < 0:
        kx, ky = ky, kx
    Sx, Sy, Sz = d[kx] / d[kz], d[ky] / d[kz], f(1) / d[kz]
    P = [v - o for v in tri]
    X = [p[kx] - Sx * p[kz] for p in P]
    Y = [p[ky] - Sy * p[kz] for p in P]
    U, V, W = X[2] * Y[1] - Y[2] * X[1], X[0] * Y[2] - Y[0] * X[2], X[1] * Y[0] - Y[1] * X[0]
    if (U < 0 or V < 0 or W < 0) and (U > 0 or V > 0 or W > 0):
        return NAN
    return (U * (Sz * P[0][kz]) + V * (Sz * P[1][kz]) + W * (Sz * P[2][kz])) * (f(1) / (U + V + W))


def test_lost_rays_have_no_distance():
    rng = np.random.default_rng(5)
    with np.errstate(all="ignore"):
        for o, d in _lost_rays():
            for _ in range(200):
                t = _distance(o, d, rng.uniform(-1, 1, (3, 3)).astype(np.float32))
                assert not (t > 0 and t < INF)


@pytest.mark.gpu
@pytest.mark.parametrize("width", [2, 4, 8])
def test_lost_rays_miss(width):
    sc = workloads.sphere_field(3, 64, 64, seed=2)
    sc.Prepare()
    rng = np.random.default_rng(3)
    rays = np.zeros((4096, 8), np.float32)
    rays[:, 0:3] = rng.uniform(0, 20, (4096, 3))
    rays[:, 4:7] = rng.standard_normal((4096, 3))
    rays[:, 7] = INF
    ctx = _native.default_context()
    base = _native.get_tuning(ctx)
    _native.set_tuning(ctx, traceBvhWidth=width)
    try:
        want, blocked = sc.native.trace(rays), sc.native.occluded(rays)
        mixed, at = rays.copy(), []
        for k, (o, d) in enumerate(_lost_rays()):
            at.append(17 + 173 * k)
            mixed[at[-1], 0:3], mixed[at[-1], 4:7] = o, d
        got, got_blocked = sc.native.trace(mixed), sc.native.occluded(mixed)
    finally:
        _native.set_tuning(ctx, **base)
    assert (got[at, 3].view(np.int32) == -1).all() and not got_blocked[at].any()
    rest = np.setdiff1d(np.arange(4096), at)
    assert np.array_equal(got[rest].view(np.uint32), want[rest].view(np.uint32))
    assert np.array_equal(got_blocked[rest], blocked[rest])


def _axis_rays(rng, n):
    """Rays with one or two direction components of either zero sign, or of a denormal size."""
    d = rng.standard_normal((n, 3)).astype(np.float32)
    small = np.array([0.0, -0.0, 1e-39, -1e-39], np.float32)
    first = rng.integers(0, 3, n)
    for axes in (first, np.where(rng.random(n) < 0.5, (first + 1) % 3, first)):
        d[np.arange(n), axes] = small[rng.integers(0, 4, n)]
    rays = np.zeros((n, 8), np.float32)
    rays[:, 0:3], rays[:, 4:7], rays[:, 7] = rng.uniform(0, 20, (n, 3)), d, INF
    return rays


@pytest.mark.gpu
@pytest.mark.parametrize("width", [2, 4, 8])
def test_axis_rays_hit_what_fp64_hits(width):
    """Primitive exact and t to a relative 1e-5 on non-degenerate rays (the repository's intersection
    criterion), and no ray along an axis falls between two triangles that share an edge."""
    from oracle import pyoracle as O
    sc = workloads.sphere_field(3, 64, 64, seed=2)
    sc.Prepare()
    rays = _axis_rays(np.random.default_rng(11), 900)
    # straight down onto the floor's diagonal (x + z = 20), outside the spheres
    x = np.array([-15, -10.5, -5, 30, 41.25, 50], np.float32)
    floor = np.zeros((len(x), 8), np.float32)
    floor[:, 0], floor[:, 1], floor[:, 2], floor[:, 5], floor[:, 7] = x, 5, 20 - x, -1, INF
    ctx = _native.default_context()
    base = _native.get_tuning(ctx)
    _native.set_tuning(ctx, traceBvhWidth=width)
    try:
        hits, occ, down = sc.native.trace(rays), sc.native.occluded(rays), sc.native.trace(floor)
    finally:
        _native.set_tuning(ctx, **base)
    ref, second = O.OracleScene.from_scene(sc).trace_brute64(rays[:, 0:3].astype(np.float64), rays[:, 4:7].astype(np.float64), with_second=True)
    t, u, v, tri = ref.T
    scale = np.maximum(np.abs(rays[:, 0:3]).max(1), 1.0)
    sure = (tri >= 0) & (np.minimum(np.minimum(u, v), 1 - u - v) >= 1e-4) & (second - t >= 1e-4 * t) & (t >= 0.05 * scale)
    assert sure.sum() >= 100  # enough rays to mean something: decided by the referee alone
    ids = np.ascontiguousarray(hits[:, 3:5]).view(np.int32)
    first = np.cumsum([0] + [m.NumFaces for m in sc.Meshes])
    assert np.array_equal(first[ids[sure, 1]] + ids[sure, 0], tri[sure].astype(np.int64))
    assert (np.abs(hits[sure, 0] - t[sure]) <= 1e-5 * t[sure]).all()
    assert np.array_equal(occ != 0, ids[:, 0] >= 0)
    assert (np.ascontiguousarray(down[:, 3:5]).view(np.int32)[:, 0] >= 0).all() and (np.abs(down[:, 0] - 6.5) <= 6.5e-5).all()
