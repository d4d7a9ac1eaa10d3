"""What this renderer is used for, as measurable cases.

Each case is one call (or the few calls that belong together) through the package's public
entry points, with what a user's program has in hand before it: the finalized scene on the
GPU, cameras, rays, the image to process.

  trace    SceneBVH's queries: one ray at a time from host code, host batches in the
           reference's traversal order, large device batches (closest hit and occlusion)
  render   one frame: previews of a few thousand paths, the Cornell box, the outdoor scene
           with its environment map, odd sizes, into device tensors and host arrays
  batch    many scenes, sizes and sample counts in one call
  diff     one optimisation step's forward and backward through torch.autograd
  views    many views of one scene: their images in one call, the gradients in another
  film     tone mapping and the file encoders on a finished image

Scenes are the procedural ones of mcrt_gb300.scenes.  A seed turns the geometry, moves the
camera, and draws the materials, rays, images and random-number seeds.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from mcrt_gb300 import TRAVERSE_FAST, TRAVERSE_REF, film, scenes
from mcrt_gb300.autograd import DiffRender
from mcrt_gb300.scene import CameraDesc, GpuScene, SceneDesc, render_adjoint_batch, render_batch

# rays traced per path (camera, bounces and next-event rays), of the order the scenes give
RAYS_PER_PATH = {"cornell": 5.0, "outdoor": 4.0, "mixed": 6.0}


def listed():
    return [
        # SceneBVH::intersect called by host code, one ray per call: all latency
        dict(name="trace_one_ray", kind="trace", scene="cornell", level=4, query="closest", order="fast", rays=1,
             where="host", spread=1.0),
        # host arrays through the reference's own traversal order: parity runs, picking, baking
        dict(name="trace_ref_host", kind="trace", scene="ball", level=5, query="closest", order="ref", rays=20011,
             where="host", spread=1.0),
        # the reference's random-ray measurement: 2 M incoherent closest hits, 1.3 M triangles
        dict(name="trace_closest_2m", kind="trace", scene="outdoor", level=8, query="closest", order="fast",
             rays=2000003, where="device", spread=1.0),
        # occlusion of points on a surface toward a sky of directions (baking, visibility)
        dict(name="trace_any_300k", kind="trace", scene="outdoor", level=6, query="any", order="fast", rays=300001,
             where="device", spread=0.3),
        # an interactive preview: a few thousand paths, latency and launches
        dict(name="render_preview", kind="render", scene="cornell", level=4, width=61, height=47, spp=1, depth=4,
             rr=-1, where="device"),
        # the Cornell box with area light and Russian roulette
        dict(name="render_cornell", kind="render", scene="cornell", level=4, width=256, height=256, spp=16, depth=8,
             rr=3, where="device"),
        # an odd-sized outdoor frame returned to host memory
        dict(name="render_outdoor_odd", kind="render", scene="outdoor", level=6, width=333, height=517, spp=5,
             depth=6, rr=-1, where="host"),
        # the headline frame: 1.3 M triangles, environment map with a sun, 67 M paths
        dict(name="render_outdoor_full", kind="render", scene="outdoor", level=8, width=1024, height=1024, spp=64,
             depth=16, rr=-1, where="device"),
        # scenes of different sizes, resolutions and sample counts in one call
        dict(name="batch_mixed", kind="batch", scenes=12, level=6, scale=0.5),
        # one optimisation step on 256 albedos and the emitter: image, then both gradients
        dict(name="diff_cornell", kind="diff", groups=256, width=512, height=512, spp=32, depth=6),
        # several views of the outdoor scene and the gradients of its 4096 albedos
        dict(name="adjoint_views", kind="views", level=8, groups=4096, views=8, width=256, height=256, spp=16, depth=8),
        # a finished frame: its .hdr file, then Reinhard tone mapping and the .ppm file
        dict(name="film_frame", kind="film", width=1023, height=767, op="reinhard"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trace", "trace", "render", "render", "render", "batch", "diff", "views", "film", "film"])
    if kind == "trace":
        order = rng.choice(["fast", "fast", "ref"])
        where = rng.choice(["host", "device"])
        return dict(kind=kind, scene=rng.choice(["cornell", "ball", "outdoor"]), level=rng.randint(3, 7),
                    query=rng.choice(["closest", "any"]), order=order,
                    rays=_log(rng, 1, 200000 if where == "host" else 2000000), where=where,
                    spread=rng.choice([0.3, 1.0]))
    if kind == "render":
        return dict(kind=kind, scene=rng.choice(["cornell", "outdoor"]), level=rng.randint(3, 7),
                    width=_log(rng, 17, 900), height=_log(rng, 17, 900), spp=_log(rng, 1, 24), depth=rng.randint(1, 16),
                    rr=rng.choice([-1, -1, 3]), where=rng.choice(["host", "device"]))
    if kind == "batch":
        return dict(kind=kind, scenes=rng.randint(2, 14), level=rng.randint(4, 6),
                    scale=round(rng.uniform(0.2, 0.6), 3))
    if kind == "diff":
        return dict(kind=kind, groups=_log(rng, 8, 1024), width=_log(rng, 33, 512), height=_log(rng, 33, 512),
                    spp=_log(rng, 2, 32), depth=rng.randint(2, 9))
    if kind == "views":
        return dict(kind=kind, level=rng.randint(5, 7), groups=_log(rng, 64, 4096), views=rng.randint(2, 8),
                    width=_log(rng, 33, 256), height=_log(rng, 33, 256), spp=_log(rng, 2, 16), depth=rng.randint(2, 9))
    return dict(kind=kind, width=_log(rng, 31, 1900), height=_log(rng, 31, 1000), op=rng.choice(["reinhard", "gamma"]))


# ---------------------------------------------------------------------------
# scenes: base geometry is made once per process, a seed turns and scales it
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _base(kind: str, level: int, groups: int = 0):
    if kind == "cornell":
        return scenes.cfg0_scene(sphere_level=level)
    if kind == "outdoor":
        return scenes.cfg1_scene(level=level)
    if kind == "ball":
        v, n = scenes.displaced_sphere(level, 1.0, 0.1, 5)
        return SceneDesc(v, np.zeros(v.shape[0], np.int32), [scenes.Material(scenes.DIFF, (0.7, 0.7, 0.7))], normals=n)
    if kind == "groups":
        return scenes.cfg4_scene(level=level, n_params=groups)[0]
    raise ValueError(kind)


def _seeded(base: SceneDesc, seed: int, turn: bool) -> SceneDesc:
    """The base scene scaled a little and, where its layout allows, turned about the vertical."""
    rng = np.random.default_rng(seed)
    a = rng.uniform(0.0, 2.0 * math.pi) if turn else 0.0
    r = np.array([[math.cos(a), 0.0, math.sin(a)], [0.0, 1.0, 0.0], [-math.sin(a), 0.0, math.cos(a)]], np.float32)
    s = np.float32(rng.uniform(0.96, 1.04))
    v = (base.vertices.reshape(-1, 3) @ r.T * s).reshape(-1, 9)
    n = (base.normals.reshape(-1, 3) @ r.T).reshape(-1, 9)
    return SceneDesc(v, base.material_ids, list(base.materials), normals=n, envmap=base.envmap, name=base.name)


def _scene(kind: str, level: int, seed: int, groups: int = 0) -> GpuScene:
    return GpuScene(_seeded(_base(kind, level, groups), seed, kind != "cornell"))


def _camera(kind: str, width: int, height: int, seed: int) -> CameraDesc:
    rng = np.random.default_rng(seed + 1)
    j = rng.uniform(-0.1, 0.1, 3)
    c = scenes.cfg1_camera(width, height) if kind == "outdoor" else scenes.cfg0_camera(width, height)
    c.origin = tuple(float(o + d) for o, d in zip(c.origin, j))
    return c


def _rays(kind: str, n: int, spread: float, seed: int) -> torch.Tensor:
    """(n, 8) rays on the GPU.  spread 1: origins all over the scene, uniform directions;
    below 1: origins near the object's surface, directions within the upper hemisphere."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    d = torch.randn((n, 3), generator=g, device="cuda")
    d = d / d.norm(dim=1, keepdim=True)
    if spread >= 1.0:
        ext = 2.0 if kind == "outdoor" else 1.0
        o = (torch.rand((n, 3), generator=g, device="cuda") * 2.0 - 1.0) * ext
    else:
        o = torch.randn((n, 3), generator=g, device="cuda")
        o = o / o.norm(dim=1, keepdim=True) * (1.0 + spread * torch.rand((n, 1), generator=g, device="cuda"))
        d[:, 1] = d[:, 1].abs()
    r = torch.empty((n, 8), device="cuda")
    r[:, 0:3] = o
    r[:, 3] = 1e-4
    r[:, 4:7] = d
    r[:, 7] = 1e30
    return r


def _mixed_jobs(case, seed):
    rng = np.random.default_rng(seed)
    gpu, cams, params = [], [], []
    # the mix is one list of scenes; a seed changes the geometry's scale, cameras and sampling
    for k, (desc, cam, p) in enumerate(_mixed_base(case["scenes"], case["level"])):
        gpu.append(GpuScene(_seeded(desc, seed * 131 + k, False)))
        w, h = (max(16, int(side * case["scale"])) for side in (cam.width, cam.height))
        cams.append(_camera("cornell", w - k % 2, h, seed * 131 + k))
        params.append(dict(spp=max(1, p["spp"] // 4), max_depth=p["max_depth"], rr_depth=-1,
                           seed=int(rng.integers(1 << 30))))
    return gpu, cams, params


@functools.lru_cache(maxsize=None)
def _mixed_base(n, level):
    return scenes.cfg2_jobs(n_scenes=n, max_level=level)


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed + 2)
    if kind == "trace":
        rays = _rays(case["scene"], case["rays"], case["spread"], seed)
        return dict(case=case, scene=_scene(case["scene"], case["level"], seed),
                    rays=rays if case["where"] == "device" else rays.cpu().numpy())
    if kind == "render":
        out = torch.empty((case["height"], case["width"], 3), device="cuda") if case["where"] == "device" else None
        return dict(case=case, scene=_scene(case["scene"], case["level"], seed),
                    camera=_camera(case["scene"], case["width"], case["height"], seed), out=out,
                    seed=int(rng.integers(1 << 30)))
    if kind == "batch":
        gpu, cams, params = _mixed_jobs(case, seed)
        outs = [torch.empty((c.height, c.width, 3), device="cuda") for c in cams]
        return dict(case=case, scenes=gpu, cameras=cams, params=params, outs=outs)
    if kind == "diff":
        albedo = rng.uniform(0.1, 0.9, (case["groups"], 3)).astype(np.float32)
        emission = rng.uniform(4.0, 17.0, (1, 3)).astype(np.float32)
        cam = _camera("cornell", case["width"], case["height"], seed)
        render = DiffRender(GpuScene(_seeded(scenes.cfg3_with_params(albedo, emission), seed, False)), cam,
                            spp=case["spp"], max_depth=case["depth"], seed=int(rng.integers(1 << 30)))
        g = torch.Generator(device="cuda").manual_seed(seed)
        return dict(case=case, render=render, albedo=torch.tensor(albedo, device="cuda", requires_grad=True),
                    emission=torch.tensor(emission, device="cuda", requires_grad=True),
                    target=torch.rand((cam.height, cam.width, 3), generator=g, device="cuda"))
    if kind == "views":
        sc = _scene("groups", case["level"], seed, case["groups"])
        albedo = rng.uniform(0.1, 0.9, (len(sc.desc.materials), 3))
        mats = [scenes.Material(m.type, tuple(float(x) for x in a) if m.albedo_param >= 0 else m.color,
                                albedo_param=m.albedo_param) for m, a in zip(sc.desc.materials, albedo)]
        sc.set_materials(mats)
        cams = scenes.fibonacci_cameras(case["views"], width=case["width"], height=case["height"])
        g = torch.Generator(device="cuda").manual_seed(seed)
        dls = [torch.randn((c.height, c.width, 3), generator=g, device="cuda") for c in cams]
        params = [dict(spp=case["spp"], max_depth=case["depth"], rr_depth=-1, seed=int(rng.integers(1 << 30)))
                  for _ in cams]
        outs = [torch.empty((c.height, c.width, 3), device="cuda") for c in cams]
        return dict(case=case, scenes=[sc] * len(cams), cameras=cams, params=params, outs=outs, dls=dls)
    # film: a frame's radiance, over the range a rendered scene has (dark corners to a sun)
    g = torch.Generator(device="cuda").manual_seed(seed)
    img = torch.rand((case["height"], case["width"], 3), generator=g, device="cuda")
    img = img * torch.exp2(torch.randn((case["height"], case["width"], 1), generator=g, device="cuda") * 2.0 - 1.0)
    dark = torch.rand((case["height"], case["width"], 1), generator=g, device="cuda") < 0.03
    return dict(case=case, img=torch.where(dark, torch.zeros_like(img), img))


def _bytes(data: bytes) -> np.ndarray:
    return np.frombuffer(data, np.uint8)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "trace":
        order = TRAVERSE_REF if case["order"] == "ref" else TRAVERSE_FAST
        if case["query"] == "any":
            return {"occluded": state["scene"].trace_any(state["rays"], order)}
        h = state["scene"].trace_closest(state["rays"], order)
        prim = h[:, 3].view(torch.int32) if case["where"] == "device" else h[:, 3].view(np.int32)
        return {"t": h[:, 0], "uv": h[:, 1:3], "prim": prim}
    if kind == "render":
        img, _ = state["scene"].render(state["camera"], spp=case["spp"], max_depth=case["depth"],
                                       rr_depth=case["rr"], seed=state["seed"], out=state["out"])
        return {"image": img}
    if kind == "batch":
        outs, _ = render_batch(state["scenes"], state["cameras"], state["params"], outs=state["outs"])
        return {"images": list(outs)}
    if kind == "diff":
        img = state["render"](state["albedo"], state["emission"])
        loss = ((img - state["target"]) ** 2).mean()
        ga, ge = torch.autograd.grad(loss, (state["albedo"], state["emission"]))
        return {"image": img.detach(), "d_albedo": ga, "d_emission": ge}
    if kind == "views":
        outs, _ = render_batch(state["scenes"], state["cameras"], state["params"], outs=state["outs"])
        ga, _, _ = render_adjoint_batch(state["scenes"], state["cameras"], state["params"], state["dls"],
                                        case["groups"], 0)
        return {"images": list(outs), "d_albedo": ga}
    hdr = film.encode(state["img"], "hdr")
    ldr = film.tonemap(state["img"].clone(), case["op"])
    return {"hdr": _bytes(hdr), "ldr": ldr, "ppm": _bytes(film.encode(ldr, "ppm"))}


def _triangles(case) -> int:
    kind = case["kind"]
    if kind == "batch":
        return sum(d.num_triangles for d, _, _ in _mixed_base(case["scenes"], case["level"]))
    if kind == "diff":
        return 12 + 20 * 4 ** 4
    return 20 * 4 ** case["level"] + (12 if case.get("scene") == "cornell" else 2)


def work(case):
    """One pass: each input read once, each output written once; for the flops, every ray
    tests the boxes of one path down a binary tree and one triangle, and nothing else."""
    kind = case["kind"]
    if kind == "film":
        px = case["width"] * case["height"]
        return {"bytes": px * (12 + 12 + 4 + 3), "flops": px * 3 * 10}
    tris = _triangles(case)
    per_ray = 24 * math.log2(tris) + 60
    if kind == "trace":
        out = 4 if case["query"] == "any" else 16
        return {"bytes": case["rays"] * (32 + out) + min(36 * tris, case["rays"] * 36 * 2),
                "flops": case["rays"] * per_ray}
    if kind == "batch":
        paths = px = 0
        for _, cam, p in _mixed_base(case["scenes"], case["level"]):
            n = int(cam.width * case["scale"]) * int(cam.height * case["scale"])
            px += n
            paths += n * max(1, p["spp"] // 4)
        return {"bytes": 76 * tris + 12 * px, "flops": paths * RAYS_PER_PATH["mixed"] * per_ray}
    n = case["width"] * case["height"] * case.get("views", 1)
    outdoor = kind == "views" or case.get("scene") == "outdoor"
    env = 12 * 1024 * 512 if outdoor else 0
    rays = n * case["spp"] * RAYS_PER_PATH["outdoor" if outdoor else "cornell"]
    back = 2 if kind in ("diff", "views") else 1
    rays *= back
    return {"bytes": 76 * tris + env + 12 * n * back + 12 * case.get("groups", 0),
            "flops": rays * per_ray}


# ---------------------------------------------------------------------------
# values in 64 bits
# ---------------------------------------------------------------------------
def _closest64(vertices, rays):
    """Closest hits by testing every triangle (Moeller-Trumbore, |det| >= 1e-6) in float64."""
    v = torch.as_tensor(vertices, device="cuda", dtype=torch.float64).reshape(-1, 3, 3)
    r = torch.as_tensor(rays, device="cuda", dtype=torch.float64)
    a, e1, e2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    t_out = torch.full((r.shape[0],), math.inf, device="cuda", dtype=torch.float64)
    uv_out = torch.zeros((r.shape[0], 2), device="cuda", dtype=torch.float64)
    step = max(1, (1 << 23) // max(1, v.shape[0]))
    for k in range(0, r.shape[0], step):
        o, d = r[k:k + step, None, 0:3], r[k:k + step, None, 4:7]
        lo, hi = r[k:k + step, None, 3], r[k:k + step, None, 7]
        p = torch.linalg.cross(d.expand(-1, v.shape[0], -1), e2.expand(d.shape[0], -1, -1))
        det = (e1 * p).sum(-1)
        inv = 1.0 / det
        s = o - a
        u = (s * p).sum(-1) * inv
        q = torch.linalg.cross(s, e1.expand(d.shape[0], -1, -1))
        w = (d * q).sum(-1) * inv
        t = (e2 * q).sum(-1) * inv
        ok = (det.abs() >= 1e-6) & (u >= 0) & (u <= 1) & (w >= 0) & (u + w <= 1) & (t > lo) & (t < hi)
        t = torch.where(ok, t, math.inf)
        best, at = t.min(dim=1)
        hit = torch.isfinite(best)
        t_out[k:k + step] = best
        uv = torch.stack([u.gather(1, at[:, None])[:, 0], w.gather(1, at[:, None])[:, 0]], 1)
        uv_out[k:k + step] = torch.where(hit[:, None], uv, 0.0)
    return t_out, uv_out


def exact(case, seed):
    kind = case["kind"]
    if kind == "trace" and case["query"] == "closest" and case["rays"] * _triangles(case) <= 1 << 30:
        state = prepare(case, seed)
        t, uv = _closest64(state["scene"].desc.vertices, state["rays"])
        return {"t": t, "uv": uv, "prim": None}
    if kind == "film":
        x = prepare(case, seed)["img"].to(torch.float64)
        if case["op"] == "gamma":
            ldr = x.clamp(0.0, 1.0) ** (1.0 / 2.2)
        else:
            # Reinhard's operator with contrast 0.77, chromatic and light adaptation 0.5 and 0
            lum = (0.299 * x[..., 0] + 0.587 * x[..., 1] + 0.114 * x[..., 2]).clamp(min=1e-7).mean()
            k = (0.5 * x.mean(dim=(0, 1)) + 0.5 * lum) ** 0.77
            ldr = x / (x + k)
        return {"hdr": None, "ldr": ldr, "ppm": None}
    return None
