"""The environment map's sampling tables equal sequential single-precision sums bit for bit: samples
drawn with the CDF entries themselves, and with the next float above them, select the texel that the
host's tables select (the first entry >= u; Sampling/PiecewiseConstant.cs:12-50), at widths and heights
around the 32 lanes that build a row."""
import ctypes

import numpy as np
import pytest

from seesharp_gb300 import EnvironmentMap, RgbImage, _native, workloads

pytestmark = pytest.mark.gpu


def _cdf(values):
    out, s = np.zeros(len(values), np.float32), np.float32(0)
    for k, v in enumerate(values):
        s = np.float32(s + v)
        out[k] = s
    if s > 0:
        out = (out / s).astype(np.float32)
    out[-1] = 1
    return out, s


@pytest.mark.parametrize("w,h", [(1, 1), (31, 2), (32, 3), (33, 5), (64, 31), (97, 33), (130, 64)])
def test_samples_select_the_sequential_tables_texel(w, h):
    rng = np.random.default_rng(w * 1000 + h)
    # distinct grey values, so that a sample's radiance names its texel; a black texel and a black row
    v = (rng.permutation(w * h).reshape(h, w) + 10).astype(np.float32) / np.float32(w * h)
    if w > 2 and h > 2:
        v[1, 1] = 0
        v[2] = 0
    img = np.repeat(v[:, :, None], 3, 2)
    lum = (np.float32(0.2126) * v + np.float32(0.7152) * v).astype(np.float32) + np.float32(0.0722) * v
    rows = [_cdf(r) for r in lum]
    marg, _ = _cdf([s for _, s in rows])
    us, want = [], []
    for _ in range(4000):
        u2 = marg[rng.integers(h)]
        u2 = np.nextafter(u2, np.float32(2)) if rng.random() < 0.5 else u2
        u2 = np.minimum(u2, np.float32(1))
        r = int(np.searchsorted(marg, u2, "left"))
        cdf = rows[r][0]
        u1 = cdf[rng.integers(w)]
        u1 = np.nextafter(u1, np.float32(2)) if rng.random() < 0.5 else u1
        u1 = np.minimum(u1, np.float32(1))
        c = int(np.searchsorted(cdf, u1, "left"))
        us.append((u1, u2))
        want.append((r, c))
    sc = workloads.env_lit_box(8, 8)
    sc.Background = EnvironmentMap(RgbImage(img))
    sc.Prepare()
    n = len(us)
    us = np.array(us, np.float32)
    dirs, pdfs, ws = np.zeros((n, 3), np.float32), np.zeros(n, np.float32), np.zeros((n, 3), np.float32)
    q, rad, qp = np.tile(np.float32([0, 1, 0]), (n, 1)), np.zeros((n, 3), np.float32), np.zeros(n, np.float32)
    p = lambda a: ctypes.c_void_p(a.ctypes.data)  # noqa: E731
    _native.check(sc.native.lib.sst_debug_envmap(sc.native.handle, n, p(us), p(dirs), p(pdfs), p(ws), p(q), p(rad), p(qp)))
    # the sample lies in the chosen cell, inside or on its edge (the relative position is in [0, 1])
    phi = np.arctan2(dirs[:, 2].astype(np.float64), dirs[:, 0]) % (2 * np.pi)
    theta = np.arccos(np.clip(dirs[:, 1].astype(np.float64), -1, 1))
    r, c = np.array(want).T
    x, y = phi / (2 * np.pi) * w, theta / np.pi * h
    dx = np.abs((x - c - 0.5 + w / 2) % w - w / 2)
    azimuth = np.sin(theta) > 1e-4  # a sample on a pole (the outer edge of the first or last row) has none
    assert (dx[azimuth] <= 0.5 + 1e-3).all() and (np.abs(y - r - 0.5) <= 0.5 + 1e-3).all()
