"""Films do not depend on the order in which a wave's paths are shaded: image sizes around the wave of
65536 paths, up to which the paths stay in queue order."""
import numpy as np
import pytest

from seesharp_gb300 import _native, workloads
from seesharp_gb300.integrators import PathTracer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", [0, 1])
@pytest.mark.parametrize("size", [(1, 1), (31, 7), (255, 257), (256, 256), (257, 256)])
def test_films_around_the_wave_that_is_ordered(size, split):
    ctx = _native.default_context()
    base = _native.get_tuning(ctx)
    sc = workloads.sphere_field(6, size[0], size[1], seed=2)
    sc.Prepare()
    films = []
    try:
        for order in (0, 1):
            for capacity in (0, 4096):  # a wave of the whole image, and waves that are never ordered
                _native.set_tuning(ctx, **dict(base, shadeOrder=order, shadeSplit=split, waveCapacity=capacity))
                pt = PathTracer(TotalSpp=1, MaxDepth=4, BaseSeed=7)
                sc.FrameBuffer.Reset()
                pt.Render(sc)
                films.append((sc.FrameBuffer.Image.data.copy(), pt.last_stats.numRays, pt.last_stats.numShadowRays))
    finally:
        _native.set_tuning(ctx, **base)
    for img, rays, shadow in films[1:]:
        assert np.array_equal(img.view(np.uint32), films[0][0].view(np.uint32))
        assert (rays, shadow) == films[0][1:]
