"""The environment map's sampling tables, read back from the kernels that build them, hold the bits of
sequential single-precision sums: every entry of the column and row tables, the row sums and the row flags,
at widths and heights around the 32 lanes that build a row, with black rows, values of very different
sizes, infinities and NaN."""
import ctypes

import numpy as np
import pytest

from seesharp_gb300 import _native

pytestmark = pytest.mark.gpu

# sst::launch_env_build(const float4* img, int w, int h, float* colCdf, float* rowMarg, int* hasCol, float* rowCdf, cudaStream_t)
BUILD = "_ZN3sst16launch_env_buildEPK6float4iiPfS3_PiS3_P11CUstream_st"


def _cdf(values):
    """Running sums in order, divided by the total when that is positive, the last set to one."""
    out = np.zeros(len(values), np.float32)
    s = np.float32(0)
    for k, v in enumerate(values):
        s = np.float32(s + v)
        out[k] = s
    if s > 0:
        out = (out / s).astype(np.float32)
    out[-1] = 1
    return out, s


@pytest.mark.parametrize("w,h", [(1, 1), (2, 33), (31, 2), (32, 32), (33, 5), (64, 31), (97, 64), (130, 65), (1025, 3)])
@pytest.mark.parametrize("kind", ["ordinary", "uneven", "special"])
def test_tables_are_the_sequential_sums(w, h, kind):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(1000 * w + h)
    img = rng.random((h, w, 4)).astype(np.float32)
    if kind != "ordinary":
        img *= np.exp(rng.uniform(-30, 30, (h, w, 1))).astype(np.float32)
        img[h // 2] = 0
    if kind == "special":
        img[0, w - 1, 1] = np.inf
        img[h - 1, 0, 2] = np.nan
    with np.errstate(all="ignore"):
        lum = (np.float32(0.2126) * img[..., 0] + np.float32(0.7152) * img[..., 1]).astype(np.float32) + np.float32(0.0722) * img[..., 2]
        rows = [_cdf(r) for r in lum]
        col, marg = np.array([c for c, _ in rows]), np.array([s for _, s in rows], np.float32)
        row, _ = _cdf(marg)
    d = torch.from_numpy(img).cuda()
    out = [torch.full(s, -7.0, device="cuda") for s in ((h, w), (h,), (h,))]
    has = torch.full((h,), -7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    fn = getattr(_native.load_library(), BUILD)
    fn.restype = None
    fn(p(d), ctypes.c_int(w), ctypes.c_int(h), p(out[0]), p(out[1]), p(has), p(out[2]), ctypes.c_void_p(None))
    torch.cuda.synchronize()
    for got, want in zip(out, (col, marg, row)):
        got = got.cpu().numpy()
        nan = np.isnan(want)
        assert np.array_equal(np.isnan(got), nan)
        assert np.array_equal(got[~nan].view(np.uint32), want[~nan].view(np.uint32))
    assert np.array_equal(has.cpu().numpy() != 0, marg != 0)
