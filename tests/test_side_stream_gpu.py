"""The second stream of a render and of its adjoint: gradients from the wavefront, whose next-event
rays and ended paths run beside the next extension rays, against the replay of one path per
thread, which runs on one stream; and calls on a stream of the caller's own, whose earlier work
they must come after."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, H, SPP, GROUPS = 33, 29, 3, 16


@pytest.fixture(scope="module")
def lit(cuda_device):
    """A parameterised Cornell box with its area light, and the same under an environment too."""
    from mcrt_gb300 import GpuScene, scenes
    rng = np.random.default_rng(6)
    desc = scenes.cfg3_with_params(rng.uniform(0.2, 0.8, (GROUPS, 3)).astype(np.float32),
                                   np.array([[17.0, 12.0, 4.0]], np.float32), sphere_level=2)
    both = dataclasses.replace(desc, envmap=scenes.sky_envmap(64, 32))
    return {"area": GpuScene(desc), "both": GpuScene(both)}, scenes.cfg0_camera(W, H)


@pytest.mark.parametrize("chunk", [0, 64, W * H * SPP - 1])
@pytest.mark.parametrize("depth", [0, 1, 2, 6])
@pytest.mark.parametrize("lights", ["area", "both"])
def test_adjoint_with_overlap_equals_the_replay_on_one_stream(lights, depth, chunk, lit):
    scenes, cam = lit
    dl = np.random.default_rng(depth).normal(size=(H, W, 3)).astype(np.float32)
    args = (cam, SPP, depth, dl, GROUPS, 1)
    want = scenes[lights].render_adjoint(*args, seed=5, schedule=1)
    got = scenes[lights].render_adjoint(*args, seed=5, path_chunk=chunk)
    for g, w in zip(got[:2], want[:2]):
        # the bound of the other comparison with the replay: the order of float sums
        assert np.linalg.norm(g - w) <= 1e-4 * np.linalg.norm(w)


def _slow(device):
    """A few milliseconds of work on the current stream."""
    import torch
    w = torch.ones((4096, 4096), device=device)
    for _ in range(12):
        w = (w @ w).clamp_(max=1.0)
    return w


@pytest.mark.parametrize("chunk", [0, 64])
def test_calls_on_a_callers_stream_come_after_its_earlier_work(chunk, lit, cuda_device):
    import torch
    scenes, cam = lit
    scene = scenes["both"]
    kw = dict(spp=SPP, max_depth=4, seed=9, path_chunk=chunk)
    want, _ = scene.render(cam, **kw)
    base = torch.tensor(np.random.default_rng(2).normal(size=(H, W, 3)).astype(np.float32), device=cuda_device)
    ga, ge, _ = scene.render_adjoint(cam, SPP, 4, base, GROUPS, 1, seed=9, path_chunk=chunk)
    out = torch.zeros((H, W, 3), device=cuda_device)
    dl = torch.zeros((H, W, 3), device=cuda_device)
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        _slow(cuda_device)
        out.fill_(7.0)  # overwritten by the render, unless it ran ahead
        scene.render(cam, out=out, **kw)
        got = out.clone()
        _slow(cuda_device)
        dl.copy_(base)  # read by the adjoint's kernels on both streams
        a, e, _ = scene.render_adjoint(cam, SPP, 4, dl, GROUPS, 1, seed=9, path_chunk=chunk)
    torch.cuda.synchronize()
    assert np.array_equal(got.cpu().numpy().view(np.int32), want.view(np.int32))
    for g, w in ((a, ga), (e, ge)):
        assert float((g - w).norm()) <= 1e-4 * float(w.norm())
