"""Ray queries give the same results however their arrays reach the device: host arrays below and above
the sizes that are read and written in place, device arrays on a 16-byte boundary and off it."""
import ctypes

import numpy as np
import pytest

from seesharp_gb300 import _native, workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene():
    sc = workloads.sphere_field(3, 64, 64, seed=4)
    sc.Prepare()
    return sc


@pytest.mark.parametrize("n", [1, 31, 33, 2048, 2049, 8192, 8193, 20001])
def test_results_do_not_depend_on_the_route(scene, n):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    rays = np.zeros((n, 8), np.float32)
    rays[:, 0:3], rays[:, 4:7], rays[:, 7] = rng.uniform(0, 20, (n, 3)), rng.standard_normal((n, 3)), np.inf
    sh = scene.native
    hits, occ = sh.trace(rays), sh.occluded(rays)
    # one ray at a time (always in place) and in chunks of 3000 (copied for closest hits)
    pick = rng.integers(0, n, min(n, 20))
    for k in pick:
        assert np.array_equal(sh.trace(rays[k:k + 1]).view(np.uint32), hits[k:k + 1].view(np.uint32))
        assert sh.occluded(rays[k:k + 1])[0] == occ[k]
    for a in range(0, n, 3000):
        assert np.array_equal(sh.trace(rays[a:a + 3000]).view(np.uint32), hits[a:a + 3000].view(np.uint32))
        assert np.array_equal(sh.occluded(rays[a:a + 3000]), occ[a:a + 3000])
    if n <= 65536:
        assert np.array_equal(sh.occluded_noalloc(rays), occ)
    assert np.array_equal(occ != 0, np.ascontiguousarray(hits[:, 3]).view(np.int32) >= 0)
    for shift in (0, 1, 2):  # floats from a 16-byte boundary
        buf = torch.zeros(n * 8 + 4, device="cuda")
        buf[shift:shift + n * 8] = torch.from_numpy(rays).cuda().reshape(-1)
        out, oc = torch.zeros((n, 12), device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        p = ctypes.c_void_p(buf.data_ptr() + 4 * shift)
        _native.check(sh.lib.sst_trace(sh.handle, p, n, ctypes.c_void_p(out.data_ptr()), _native.SST_MEM_DEVICE))
        _native.check(sh.lib.sst_occluded(sh.handle, p, n, ctypes.c_void_p(oc.data_ptr()), _native.SST_MEM_DEVICE))
        assert np.array_equal(out.cpu().numpy().view(np.uint32), hits.view(np.uint32)) and np.array_equal(oc.cpu().numpy(), occ)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 257, 4099])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])  # floats from a 16-byte boundary
def test_device_hits_on_any_boundary(scene, n, shift):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    rays = np.zeros((n, 8), np.float32)
    rays[:, 0:3], rays[:, 4:7], rays[:, 7] = rng.uniform(0, 20, (n, 3)), rng.standard_normal((n, 3)), np.inf
    sh = scene.native
    hits = sh.trace(rays)
    d = torch.from_numpy(rays).cuda()
    out = torch.full((12 * n + 8,), 7.0, device="cuda")
    torch.cuda.synchronize()
    _native.check(sh.lib.sst_trace(sh.handle, ctypes.c_void_p(d.data_ptr()), n, ctypes.c_void_p(out.data_ptr() + 4 * shift), _native.SST_MEM_DEVICE))
    o = out.cpu().numpy()
    assert np.array_equal(o[shift:shift + 12 * n].view(np.uint32), hits.reshape(-1).view(np.uint32))
    assert np.all(o[:shift] == 7.0) and np.all(o[shift + 12 * n:] == 7.0)
