"""The streamed traversal: a ray's answer does not depend on the batch it is traced in, on its
place in the batch or on which lane took it, so every batch size must give, ray by ray, the
bits of any other; closest-hit and any-hit queries of one ray agree on whether it hits."""
import numpy as np
import pytest

from conftest import golden
from parity import classify

pytestmark = pytest.mark.gpu

# one ray, a warp's batch and its edges, a block, more batches than a block has warps, ragged
SIZES = [1, 2, 31, 32, 33, 127, 128, 129, 1023, 20011]


def _rays(n):
    """Rays of very different lengths side by side: incoherent, short segments, misses, an
    axis-parallel direction, a direction that is not normalised."""
    rng = np.random.default_rng(11)
    r = np.zeros((n, 8), np.float32)
    r[:, 0:3] = rng.uniform(-1.5, 1.5, (n, 3))
    d = rng.normal(size=(n, 3))
    r[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r[:, 3], r[:, 7] = 1e-4, 1e30
    r[1::7, 7] = 0.05
    r[2::7, 0:3] += 50.0
    r[3::7, 4:7] = (0.0, -1.0, 0.0)
    r[4::7, 4:7] *= 3.0
    return r


@pytest.fixture(scope="module")
def scene(cuda_device):
    from mcrt_gb300 import GpuScene, scenes
    return GpuScene(scenes.cfg1_scene(level=5))


@pytest.mark.parametrize("n", SIZES)
def test_batch_size_and_order_change_no_ray(n, scene):
    rays = _rays(SIZES[-1])
    whole = scene.trace_closest(rays)
    occ = scene.trace_any(rays)
    assert np.array_equal(occ != 0, whole[:, 3].view(np.int32) >= 0)
    order = np.random.default_rng(n).permutation(rays.shape[0])[:n]
    part = scene.trace_closest(rays[order])
    assert np.array_equal(part.view(np.int32), whole[order].view(np.int32))
    assert np.array_equal(scene.trace_any(rays[order]), occ[order])


def test_streamed_hits_match_the_reference_tree(cuda_device):
    """Against SplitBVH's own hits, by the parity rule of the other traversal tests."""
    from parity import fixture_scene
    from mcrt_gb300 import GpuScene
    fx = golden("ref_traverse_sphere5.npz")
    out = GpuScene(fixture_scene(fx)).trace_closest(fx["rays_bounce"])
    bad, _ = classify(fx["verts"], fx["rays_bounce"], fx["t_bounce"], fx["prim_bounce"], out[:, 0],
                      out[:, 3].view(np.int32))
    assert not bad.any()


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("depth", [0, 1, 2, 7])
@pytest.mark.parametrize("chunk", [0, 33 * 29 * 3, 33 * 29 * 3 - 1, 64])
def test_admission_and_overlap_change_no_pixel(chunk, depth, graph, cuda_device):
    """The frame whose paths are all admitted at once (as many slots as paths, and the default),
    one slot short of that, and with 64 slots, against the wave schedule, which runs every
    kernel after the other: the same bits, for odd and even numbers of iterations.  Both lights."""
    import dataclasses
    from mcrt_gb300 import GpuScene, scenes
    desc = scenes.cfg0_scene(sphere_level=2)
    cam = scenes.cfg0_camera(33, 29)
    both = dataclasses.replace(desc, envmap=scenes.sky_envmap(64, 32))
    for d in (desc, both):
        sc = GpuScene(d)
        kw = dict(spp=3, max_depth=depth, seed=21)
        want, sw = sc.render(cam, schedule=1, **kw)
        got, sg = sc.render(cam, schedule=0, path_chunk=chunk, use_graph=graph, **kw)
        assert np.array_equal(got.view(np.int32), want.view(np.int32))
        assert sg["rays"] == sw["rays"] and sg["paths"] == 33 * 29 * 3
        if chunk == 0 and not graph:
            assert sg["waves"] == depth + 1


@pytest.mark.parametrize("chunk", [1, 127, 129, 511, 513, 0])
@pytest.mark.parametrize("kind", ["environment", "area", "both"])
def test_light_kinds_alone_and_beside_the_others(kind, chunk, cuda_device):
    """A scene with one kind of light keeps two next-event results per path, one with both (or a
    batch that has both) four: the same image alone as in a batch beside the other kinds, with
    queues around a block and around a sorted window (path_chunk paths in flight).  The bound is
    that of the other batch test: the builds may round differently."""
    import dataclasses
    from mcrt_gb300 import GpuScene, render_batch, scenes
    area = scenes.cfg0_scene(sphere_level=1)
    descs = {"area": (area, scenes.cfg0_camera(13, 11)),
             "environment": (scenes.cfg1_scene(level=2, env_size=(64, 32)), scenes.cfg1_camera(13, 11)),
             "both": (dataclasses.replace(area, envmap=scenes.sky_envmap(64, 32)), scenes.cfg0_camera(13, 11))}
    p = dict(spp=1 if chunk == 1 else 4, max_depth=4, rr_depth=2, seed=17, path_chunk=chunk)
    names = [kind] + [k for k in descs if k != kind]
    gs = {k: GpuScene(descs[k][0]) for k in names}
    alone, _ = gs[kind].render(descs[kind][1], **p)
    outs, _ = render_batch([gs[k] for k in names], [descs[k][1] for k in names], [p] * 3)
    assert alone.max() > 0
    np.testing.assert_allclose(outs[0], alone, rtol=1e-5, atol=1e-6)
