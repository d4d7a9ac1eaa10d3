"""What a render leaves behind when it returns: nothing.  Every operation it queued, on the caller's
stream and on its own second stream, has to come before something the host waited for; otherwise
the next call on the same working block meets work of the last one.  On the CPU, over a stand-in
for the CUDA runtime that keeps a clock per stream (fake_cuda)."""
import numpy as np
import pytest

import fake_cuda


@pytest.fixture(scope="module")
def built(tmp_path_factory):
    return fake_cuda.build(str(tmp_path_factory.mktemp("fake")))


@pytest.fixture
def cuda(built, monkeypatch):
    return fake_cuda.Fake(built, monkeypatch)


def _scene():
    from mcrt_gb300 import GpuScene, scenes
    return GpuScene(scenes.cfg0_scene(sphere_level=1)), scenes.cfg0_camera(16, 12)


@pytest.mark.parametrize("chunk", [0, 64])  # all paths admitted at once; admitted as paths end
@pytest.mark.parametrize("mode", ["stream", "graph", "stages", "waves", "paths", "adjoint"])
def test_a_render_returns_with_nothing_queued(mode, chunk, cuda):
    scene, cam = _scene()
    paths = 16 * 12 * 2
    cuda.polls_read(paths)  # every path has ended when the counter is first read
    for _ in range(2):
        kw = dict(spp=2, max_depth=3, path_chunk=chunk)
        if mode == "adjoint":
            scene.render_adjoint(cam, 2, 3, np.zeros((12, 16, 3), np.float32), 1, 1, path_chunk=chunk)
        else:
            scene.render(cam, use_graph=mode == "graph", profile=1 if mode == "stages" else 0,
                         schedule={"waves": 1, "paths": 2}.get(mode, 0), **kw)
        assert cuda.kernels()
        assert cuda.lib.fake_pending() == 0
        assert cuda.lib.fake_nulls() == 0
        assert cuda.lib.fake_open_captures() == 0
