"""Host code after a CUDA call failed: the error is returned, nothing half made is kept, and the next
call works.  On the CPU, over a stand-in for the CUDA runtime whose calls fail on request
(fake_cuda)."""
import numpy as np
import pytest

import fake_cuda
from mcrt_gb300 import McrtError


@pytest.fixture(scope="module")
def built(tmp_path_factory):
    return fake_cuda.build(str(tmp_path_factory.mktemp("fake")))


@pytest.fixture
def cuda(built, monkeypatch):
    return fake_cuda.Fake(built, monkeypatch)


def _scene():
    from mcrt_gb300 import GpuScene, scenes
    return GpuScene(scenes.cfg0_scene(sphere_level=1)), scenes.cfg0_camera(16, 12)


KW = dict(spp=2, max_depth=3)
PATHS = 16 * 12 * 2
INVALID_VALUE, OUT_OF_MEMORY = 1, 2


@pytest.mark.parametrize("function", ["cudaStreamWaitEvent", "cudaLaunchKernel", "cudaEventRecord"])
@pytest.mark.parametrize("nth", [1, 2, 3, 4])
def test_a_capture_that_fails_is_ended(function, nth, cuda):
    """A call that fails while the iterations are captured fails the render; the capture, which the
    workspace's side stream has joined, is ended, and the next render runs."""
    scene, cam = _scene()
    cuda.polls_read(PATHS)
    # calls before the capture: two kernels, one event
    before = {"cudaLaunchKernel": 2, "cudaEventRecord": 1}.get(function, 0)
    cuda.fail(function, before + nth, INVALID_VALUE)
    with pytest.raises(McrtError):
        scene.render(cam, use_graph=True, path_chunk=64, **KW)
    assert cuda.lib.fake_fails_left() == 0
    assert cuda.lib.fake_open_captures() == 0
    for graph in (False, True):
        scene.render(cam, use_graph=graph, path_chunk=64, **KW)
        assert cuda.lib.fake_pending() == 0


def _render(scene, cam, adjoint):
    if adjoint:
        scene.render_adjoint(cam, 2, 3, np.zeros((12, 16, 3), np.float32), 1, 1, path_chunk=64)
    else:
        scene.render(cam, path_chunk=64, **KW)


@pytest.mark.parametrize("adjoint", [False, True])
def test_a_failed_render_does_not_fail_the_next(adjoint, cuda):
    """The runtime keeps the error of a failed allocation; the next render's check of its own
    launches must not report it."""
    scene, cam = _scene()
    cuda.polls_read(PATHS)
    cuda.fail("cudaMalloc", 1, OUT_OF_MEMORY)  # the image's or the gradients' device copy
    with pytest.raises(McrtError):
        _render(scene, cam, adjoint)
    _render(scene, cam, adjoint)


@pytest.mark.parametrize("adjoint", [False, True])
@pytest.mark.parametrize("function,nth", [("cudaMalloc", k) for k in range(1, 9)] + [("cudaHostAlloc", 1)] +
                         [("cudaStreamCreateWithFlags", 1), ("cudaEventCreateWithFlags", 1),
                          ("cudaEventCreateWithFlags", 2)])
def test_a_working_block_that_could_not_be_made_whole_is_completed(function, nth, adjoint, cuda):
    """Each allocation of the first render on a device fails in turn: the render reports it, and the
    next one makes what is missing (no null pointer, stream or event reaches the runtime)."""
    scene, cam = _scene()
    cuda.polls_read(PATHS)
    cuda.fail(function, nth, OUT_OF_MEMORY)
    with pytest.raises(McrtError):
        _render(scene, cam, adjoint)
    assert cuda.lib.fake_fails_left() == 0
    _render(scene, cam, adjoint)
    assert cuda.lib.fake_nulls() == 0
    assert cuda.lib.fake_pending() == 0


def test_tone_mapping_without_kept_scratch_uses_its_own(cuda):
    """The host thread's kept scratch cannot be allocated: Reinhard takes a smaller buffer of its
    own and the call succeeds (the failed allocation's error is not taken for a launch's)."""
    from mcrt_gb300 import film
    img = np.ones((64, 64, 3), np.float32)
    cuda.fail("cudaMalloc", 2, OUT_OF_MEMORY)  # after the image's device copy
    film.tonemap(img, "reinhard")
    assert cuda.lib.fake_fails_left() == 0
    assert len(cuda.kernels()) == 4
    assert cuda.lib.fake_pending() == 0


def test_a_failed_host_trace_does_not_fail_the_next(cuda):
    scene, _ = _scene()
    rays = np.zeros((3, 8), np.float32)
    cuda.fail("cudaMalloc", 1, OUT_OF_MEMORY)  # the kept scratch
    with pytest.raises(McrtError):
        scene.trace_closest(rays)
    assert cuda.lib.fake_fails_left() == 0
    scene.trace_closest(rays)
    assert cuda.lib.fake_pending() == 0
