"""Which kernel a ray batch takes: the streamed traversal only where some warp gets a second batch
of 32 rays; below, and in the reference's order, one batch per warp.  On the CPU, over a stand-in
for the CUDA runtime (152 SMs, four resident blocks of 128 threads of any kernel)."""
import re

import numpy as np
import pytest

import fake_cuda

LANES = 152 * 4 * 128


@pytest.fixture(scope="module")
def built(tmp_path_factory):
    return fake_cuda.build(str(tmp_path_factory.mktemp("fake")))


@pytest.fixture
def cuda(built, monkeypatch):
    return fake_cuda.Fake(built, monkeypatch)


@pytest.mark.parametrize("query", ["closest", "any"])
@pytest.mark.parametrize("n", [1, 32, 33, LANES, LANES + 1, 3 * LANES])
def test_a_batch_streams_only_when_a_warp_gets_a_second_one(n, query, cuda):
    from mcrt_gb300 import TRAVERSE_FAST, TRAVERSE_REF, GpuScene, scenes
    scene = GpuScene(scenes.cfg0_scene(sphere_level=1))
    trace = scene.trace_closest if query == "closest" else scene.trace_any
    rays = np.zeros((n, 8), np.float32)
    for traverse in (TRAVERSE_FAST, TRAVERSE_REF):
        cuda.kernels()
        trace(rays, traverse)
        name, = cuda.kernels()
        any_hit, mode, stream = re.search(r"k_traceILb([01])ELi([01])ELi\d+ELi\d+ELb([01])E", name).groups()
        assert any_hit == str(int(query == "any")) and mode == str(int(traverse == TRAVERSE_REF))
        assert stream == str(int(traverse == TRAVERSE_FAST and n > LANES))
        assert cuda.lib.fake_pending() == 0
