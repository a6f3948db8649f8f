"""sst_trace_light_paths writes the same vertices as records (host or device memory) and as planes (all
floats, then all integers), which is the form the Python binding reads."""
import ctypes

import numpy as np
import pytest

from seesharp_gb300 import _native, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,depth", [(1, 1), (33, 3), (4097, 6)])
def test_records_equal_planes(n, depth):
    torch = pytest.importorskip("torch")
    sc = workloads.sphere_field(2, 32, 32, seed=6)
    sc.Prepare()
    sh = sc.native
    floats, ints, lengths, _ = sh.trace_light_paths(77, 2, n, depth)
    assert floats.shape == (n, depth + 1, 16) and ints.shape == (n, depth + 1, 6) and ints.dtype == np.int32
    assert floats.flags["C_CONTIGUOUS"] and ints.flags["C_CONTIGUOUS"] and (lengths >= 1).all()
    raw = np.full((n, depth + 1, 22), np.nan, np.float32)
    ln = np.zeros(n, np.int32)
    dev = torch.full((n, depth + 1, 22), float("nan"), device="cuda")
    dl = torch.zeros(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    stats = _native.SstRenderStats()
    for v, l, mem in ((raw.ctypes.data, ln.ctypes.data, _native.SST_MEM_HOST), (dev.data_ptr(), dl.data_ptr(), _native.SST_MEM_DEVICE)):
        _native.check(sh.lib.sst_trace_light_paths(sh.handle, 77, 2, n, depth, ctypes.c_void_p(v), ctypes.c_void_p(l), mem, ctypes.byref(stats)))
    for got, gl in ((raw, ln), (dev.cpu().numpy(), dl.cpu().numpy())):
        assert np.array_equal(gl, lengths)
        assert np.array_equal(got[..., :16].view(np.uint32), floats.view(np.uint32))
        assert np.array_equal(np.ascontiguousarray(got[..., 16:]).view(np.int32), ints)
