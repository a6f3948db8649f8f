"""Films do not depend on how a render's waves are launched: captured graphs or kernel by kernel, on two
sets of buffers or one, shaded in order or in queue order.  Every render has a context of its own, whose
waves have the capacity asked for (a context's buffers only grow), and the number of launches shows the
route that it took."""
import numpy as np
import pytest

from seesharp_gb300 import PathTracer, _native, workloads

pytestmark = pytest.mark.gpu

DEPTH = 4
W, H = 320, 240  # more paths than a wave of CAPACITY, which is more than the waves that stay in queue order
CAPACITY = 70000


def _render(monkeypatch, width, height, spp, capacity, order=1, **env):
    contexts = {}
    monkeypatch.setattr(_native, "_contexts", contexts)
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    sc = workloads.cornell_box(width, height)
    sc.Prepare()
    try:
        _native.set_tuning(sc.native.ctx, waveCapacity=capacity, shadeOrder=order)
        pt = PathTracer(TotalSpp=spp, MaxDepth=DEPTH, BaseSeed=11)
        pt.Render(sc)
        fb = sc.FrameBuffer
        film = [fb.Image.data.copy()] + [fb.layers[k].Image.data.copy() for k in sorted(fb.layers)]
        return film, pt.last_stats.numKernelLaunches, (pt.last_stats.numRays, pt.last_stats.numShadowRays)
    finally:
        sc.Dispose()
        for c in contexts.values():
            c.close()
        for k in env:
            monkeypatch.delenv(k)


def _same(a, b):
    assert len(a[0]) == len(b[0]) >= 3 and a[2] == b[2]
    for x, y in zip(a[0], b[0]):
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32))


# launches of a wave: camera, then closest hits, shade order, shade and shadow rays per bounce, then the film
# fold (and, on two sets, the advance of the set's wave index)
ORDERED, QUEUED = 4 * DEPTH, 3 * DEPTH


@pytest.mark.parametrize("spp,graphs", [(1, False), (3, False), (8, True), (9, True)])
def test_films_of_captured_and_direct_waves(monkeypatch, spp, graphs):
    waves = -(-W * H * spp // CAPACITY)
    assert 2 <= waves and (waves >= 8) == graphs and W * H * spp % CAPACITY <= 65536
    got = _render(monkeypatch, W, H, spp, CAPACITY)
    # a captured wave has the kernels of a full one; launched directly, the last one is small enough for queue order
    assert got[1] == waves * (ORDERED + 3) - (0 if graphs else DEPTH)
    plain = _render(monkeypatch, W, H, spp, CAPACITY, SST_GRAPH="0")
    assert plain[1] == waves * (ORDERED + 2) - DEPTH
    one = _render(monkeypatch, W, H, spp, CAPACITY, SST_WAVES_IN_FLIGHT="1")
    assert one[1] == waves * (ORDERED + 2)
    whole = _render(monkeypatch, W, H, spp, 1 << 21)
    assert whole[1] == ORDERED + 2
    for other in (plain, one, whole):
        _same(got, other)


@pytest.mark.parametrize("width,height", [(256, 256), (257, 256)])
def test_films_of_ordered_and_queued_waves(monkeypatch, width, height):
    ordered = width * height > 65536
    got = _render(monkeypatch, width, height, 1, 1 << 21)
    assert got[1] == (ORDERED if ordered else QUEUED) + 2
    never = _render(monkeypatch, width, height, 1, 1 << 21, order=0)
    assert never[1] == QUEUED + 2
    small = _render(monkeypatch, width, height, 1, 16384)  # 4 or 5 waves, none of them ordered
    assert small[1] == -(-width * height // 16384) * (QUEUED + 3)
    for other in (never, small):
        _same(got, other)
