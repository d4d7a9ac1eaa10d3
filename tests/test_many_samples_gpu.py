"""Pixels with many samples: the wavefront adds a pixel's samples in order, 32 at a time, from a ring
that wraps.  The same image as the plain path tracer, which adds them one after another from a
straight array, at sample counts around multiples of 32, with all paths admitted at once and with
64 in flight (the ring is then shorter than the frame and wraps inside a pixel)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=["area", "environment"])
def scene(request, cuda_device):
    from mcrt_gb300 import GpuScene, scenes
    if request.param == "area":
        return GpuScene(scenes.cfg0_scene(sphere_level=2)), scenes.cfg0_camera
    return GpuScene(scenes.cfg1_scene(level=3, env_size=(64, 32))), scenes.cfg1_camera


@pytest.mark.parametrize("chunk", [0, 64])
@pytest.mark.parametrize("spp", [1, 2, 31, 32, 33, 63, 64, 65, 96, 1000, 4097])
@pytest.mark.parametrize("size", [(1, 1), (5, 3)])
def test_samples_are_added_in_order_from_the_ring(size, spp, chunk, scene):
    gpu, camera = scene
    kw = dict(spp=spp, max_depth=3, seed=spp)
    want, _ = gpu.render(camera(*size), schedule=2, **kw)
    got, _ = gpu.render(camera(*size), path_chunk=chunk, **kw)
    assert np.array_equal(got.view(np.int32), want.view(np.int32))
