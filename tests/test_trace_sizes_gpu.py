"""Ray batches on both sides of the line between one batch per warp and the streamed traversal: a
ray's answer has the same bits in every batch it is traced in, on either side, from host and from
device arrays, and closest-hit and any-hit queries agree on whether it hits."""
import numpy as np
import pytest

from test_stream_gpu import _rays

pytestmark = pytest.mark.gpu

LARGE = 420_001  # more rays than the GPU holds lanes, whatever the kernel
# the resident lanes of the closest-hit and any-hit kernels on 152 SMs, one more, and well below
SIZES = [1, 20_011, 155_648, 155_649, 194_560, 194_561]


@pytest.fixture(scope="module", params=["outdoor", "one triangle"])
def traced(request, cuda_device):
    from mcrt_gb300 import GpuScene, scenes
    from mcrt_gb300.scene import DIFF, Material, SceneDesc
    if request.param == "outdoor":
        desc = scenes.cfg1_scene(level=5, env_size=(16, 8))
    else:
        desc = SceneDesc(np.array([[-1, -1, 0, 1, -1, 0, 0, 1, 0]], np.float32), np.zeros(1, np.int32),
                         [Material(DIFF)])
    scene = GpuScene(desc)
    rays = _rays(LARGE)
    return scene, rays, scene.trace_closest(rays), scene.trace_any(rays)


@pytest.mark.parametrize("where", ["host", "device"])
@pytest.mark.parametrize("n", SIZES)
def test_both_sides_of_the_line_give_the_same_bits(n, where, traced):
    import torch
    scene, rays, whole, occ = traced
    assert np.array_equal(occ != 0, whole[:, 3].view(np.int32) >= 0) and occ.any() and not occ.all()
    order = np.random.default_rng(n).permutation(LARGE)[:n]
    part = rays[order]
    if where == "device":
        part = torch.tensor(part, device="cuda")
        closest, hit = scene.trace_closest(part).cpu().numpy(), scene.trace_any(part).cpu().numpy()
    else:
        closest, hit = scene.trace_closest(part), scene.trace_any(part)
    assert np.array_equal(closest.view(np.int32), whole[order].view(np.int32))
    assert np.array_equal(hit, occ[order])
