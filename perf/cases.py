"""What the performance of this framework is measured on: calls of its public
API as a user's program makes them, over the sizes and options of the
benchmark configurations (wavefrontpathtracing_gb300/scenes.py).

A case is a dict of plain values with its family in "kind":

  frame    a rendered frame: Renderer.render, then the image to the host; with
           "rebuild" the scene is submitted and its TLAS built again first, as
           an interactive renderer does every frame (the reference's loop)
  pick     a few rays from host memory through Renderer.trace
  trace    a ray set on the device through Renderer.trace_device
  blas     one BLAS build through Renderer.bvh_build
  tlas     one TLAS build through Renderer.tlas_build
  adjoint  image-loss gradients through Renderer.adjoint
  batch    many scenes in one launch through Batch.render

Meshes depend on the case alone and are made once per process; what changes
with the seed is what changes from call to call in use: transforms, materials,
cameras, rays, textures, random numbers, loss gradients, vertex positions of a
mesh that is rebuilt.
"""
import functools
import math

import numpy as np
import torch

from wavefrontpathtracing_gb300 import Batch, Renderer, scenes
from wavefrontpathtracing_gb300.abi import (BSDF_DIELECTRIC, BSDF_LAMBERT, BSDF_METAL, bvh_instance_dtype,
                                            material_ext_dtype, ray_dtype)

BVH = dict(interval_count=16, max_leaf_prims=4)   # the benchmark configurations' builder options
FLT_MAX = float(np.finfo(np.float32).max)


# ------------------------------------------------------------------- the cases

def listed():
    return [
        # a click in a viewport or a handful of line-of-sight checks: the smallest call, all latency
        dict(name="pick_64", kind="pick", rays=64, instances=96, freq=16, any_hit=False),
        # the plain configuration: one sample of a 256 x 256 Lambert room
        dict(name="frame_small", kind="frame", scene="box", width=256, height=256, spp=1, bounces=4, nee=False, rr=99,
             instances=0, detail=1.0, metric=0, bounds=0, rebuild=False, textured=False, ldr=False, view_mode=0),
        # a textured room with every material under an environment map, odd sizes, written out as 8-bit
        dict(name="frame_textured", kind="frame", scene="mixed", width=613, height=377, spp=4, bounces=8, nee=True,
             rr=3, instances=0, detail=1.0, metric=0, bounds=0, rebuild=False, textured=True, ldr=True, view_mode=0),
        # the interactive loop: 300 moving instances resubmitted, TLAS rebuilt, one sample, 8-bit image
        dict(name="frame_interactive", kind="frame", scene="instanced", width=1280, height=720, spp=1, bounces=4,
             nee=True, rr=3, instances=300, detail=0.5, metric=3, bounds=1, rebuild=True, textured=False, ldr=True,
             view_mode=0),
        # the headline configuration: 1,024 instances of 8 meshes of 50k-500k triangles, 1080p, 16 samples
        dict(name="frame_instanced_1080p", kind="frame", scene="instanced", width=1920, height=1080, spp=16, bounces=8,
             nee=True, rr=3, instances=1024, detail=1.0, metric=3, bounds=1, rebuild=False, textured=False, ldr=False,
             view_mode=0),
        # shadow / visibility queries of a camera's rays against a triangle soup, an odd count
        dict(name="trace_any_coherent", kind="trace", triangles=500_000, rays=1_000_003, coherent=True, any_hit=True,
             reorder=False, layout=0),
        # the traversal micro-benchmark's hard half: random rays, closest hit, traced in origin order
        dict(name="trace_closest_incoherent", kind="trace", triangles=2_000_000, rays=1 << 22, coherent=False,
             any_hit=False, reorder=True, layout=0),
        # the plain configuration's sphere, as an editor rebuilds a mesh that was edited
        dict(name="blas_20480", kind="blas", freq=32),
        # the instanced configuration's largest mesh
        dict(name="blas_499280", kind="blas", freq=158),
        # the reference's own TLAS (its builder's default metric) over the instanced configuration's 1,025 instances
        dict(name="tlas_1025", kind="tlas", instances=1025, metric=0),
        # the differentiable configuration: 512 x 512, 64 samples, depth 6, per-triangle albedo
        dict(name="adjoint_512", kind="adjoint", width=512, height=512, spp=64, bounces=6, nee=False, rr=99,
             subdivision=5),
        # the batched configuration at a sixth of its scenes: uneven triangle counts, resolutions and samples
        dict(name="batch_11", kind="batch", scenes=11, tri_lo=1_000, tri_hi=200_000, max_side=512, bounces=6),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "pick", "trace", "trace", "blas", "tlas", "adjoint", "batch"])
    if kind == "pick":
        return dict(kind=kind, rays=_log(rng, 1, 4096), instances=_log(rng, 1, 300), freq=_log(rng, 2, 32),
                    any_hit=rng.random() < 0.5)
    if kind == "trace":
        coherent = rng.random() < 0.5
        return dict(kind=kind, triangles=_log(rng, 1_000, 2_000_000), rays=_log(rng, 10_000, 1 << 22),
                    coherent=coherent, any_hit=rng.random() < 0.5, reorder=rng.random() < (0.2 if coherent else 0.7),
                    layout=rng.choice([0, 0, 0, 1]))
    if kind == "blas":
        return dict(kind=kind, freq=_log(rng, 2, 158))
    if kind == "tlas":
        metric = rng.randrange(4)
        return dict(kind=kind, instances=_log(rng, 2, 1500 if metric < 2 else 32768), metric=metric)
    if kind == "adjoint":
        side, spp = _log(rng, 32, 512), _log(rng, 1, 32)
        nee = rng.random() < 0.5
        return dict(kind=kind, width=side, height=max(1, side - rng.randrange(16)), spp=spp, bounces=rng.randint(1, 6),
                    nee=nee, rr=rng.choice([3, 99]), subdivision=rng.randint(1, 5))
    if kind == "batch":
        return dict(kind=kind, scenes=_log(rng, 1, 12), tri_lo=1_000, tri_hi=_log(rng, 2_000, 200_000),
                    max_side=rng.choice([64, 128, 256, 512]), bounces=rng.randint(1, 8))
    scene = rng.choice(["box", "mixed", "instanced", "instanced"])
    width = _log(rng, 64, 1920)
    big = scene == "instanced"
    case = dict(kind=kind, scene=scene, width=width, height=max(1, width * 9 // 16 - rng.randrange(8)),
                spp=_log(rng, 1, 16), bounces=rng.randint(1, 8), nee=rng.random() < 0.7, rr=rng.choice([3, 99]),
                instances=_log(rng, 8, 1024) if big else 0, detail=rng.choice([0.1, 0.25, 0.5]) if big else 1.0,
                metric=rng.choice([2, 3, 3]) if big else 0, bounds=rng.randrange(2) if big else 0,
                rebuild=rng.random() < 0.5, textured=scene == "mixed" and rng.random() < 0.5, ldr=rng.random() < 0.5,
                view_mode=0)
    if rng.random() < 0.1:   # the guide images of a denoiser: albedo, world normal, depth
        case.update(view_mode=rng.choice([6, 10, 11]), spp=1)
    return case


# ---------------------------------------------------------------------- meshes

@functools.lru_cache(maxsize=None)
def _sphere(freq, seed):
    return scenes.displaced_icosphere(freq, seed=seed, amplitude=0.1)


@functools.lru_cache(maxsize=None)
def _soup(n):
    return scenes.triangle_soup(n)


@functools.lru_cache(maxsize=None)
def _room(kind, subdivision):
    return scenes.box_scene(8, 8, subdivision=subdivision) if kind == "box" else scenes.mixed_box_scene(8, 8)


@functools.lru_cache(maxsize=None)
def _batch(count, lo, hi, max_side):
    return scenes.batch_scenes(count=count, tri_range=(lo, hi),
                               resolutions=tuple(s for s in (64, 128, 256, 512) if s <= max_side))


def _with_uv(tris):
    """The same triangles with a planar uv mapping (the procedural meshes have none)."""
    t = tris.copy()
    for v in ("v0", "v1", "v2"):
        p = t[v]["position"]
        t[v]["uv"] = np.stack([p[:, 0] * 2.0 + p[:, 2], p[:, 1] * 2.0 - p[:, 2]], axis=1)
    return t


# ----------------------------------------------------------------- scene parts

def _rotations(rng, n):
    """n uniform random rotations (unit quaternions)."""
    q = rng.normal(size=(n, 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    x, y, z, w = q.T
    m = np.empty((n, 3, 3))
    m[:, 0] = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)], axis=1)
    m[:, 1] = np.stack([2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)], axis=1)
    m[:, 2] = np.stack([2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], axis=1)
    return m


def _transforms(rng, n):
    """Random rotation, uniform scale in [0.5, 2], translation in a 100^3 box."""
    t = np.zeros((n, 4, 4))
    t[:, :3, :3] = _rotations(rng, n) * rng.uniform(0.5, 2.0, size=(n, 1, 1))
    t[:, :3, 3] = rng.uniform(0.0, 100.0, size=(n, 3))
    t[:, 3, 3] = 1.0
    return t


def _materials(rng, n):
    """60 % Lambert, 25 % metal, 15 % dielectric."""
    m = np.zeros(n, dtype=material_ext_dtype)
    u = rng.random(n)
    m["bsdf"] = np.where(u < 0.60, BSDF_LAMBERT, np.where(u < 0.85, BSDF_METAL, BSDF_DIELECTRIC))
    m["ior"] = 1.5
    base = rng.uniform(0.2, 0.9, size=(n, 3))
    base[u >= 0.85] = 1.0
    m["base"]["base_color_factor"] = base
    m["base"]["roughness_factor"] = rng.uniform(0.0, 0.5, size=n)
    return m


def _instanced(r, case, rng):
    """(mesh ids, transforms, materials): the instanced configuration's
    spheres and light, the frequencies scaled by "detail"."""
    freqs = [max(2, int(round(f * case["detail"]))) for f in scenes.INSTANCED_FREQS] * 2
    ids = [r.create_mesh_from_triangles(_sphere(f, 11 + k), **BVH) for k, f in enumerate(freqs)]
    light = r.create_mesh_from_triangles(scenes.quad((30.0, 110.0, 30.0), (40.0, 0, 0), (0, 0, 40.0)), **BVH)
    n = case["instances"]
    mesh = np.array([ids[k % len(ids)] for k in range(n)] + [light], dtype=np.uint32)
    t = np.concatenate([_transforms(rng, n), np.eye(4)[None]])
    m = _materials(rng, n + 1)
    m[n] = scenes.material(base=(0.8, 0.8, 0.8), emissive=(1.0, 0.95, 0.9), strength=60.0)
    return mesh, t.astype(np.float32), m


def _room_instances(r, case, rng, textures):
    """The box or mixed-material room with seeded colours, textured when asked."""
    desc = _room(case["scene"], case.get("subdivision", 5))
    meshes = [_with_uv(t) for t in desc.meshes] if textures else desc.meshes
    ids = [r.create_mesh_from_triangles(t, **BVH) for t in meshes]
    mesh = np.array([ids[i] for i, _, _ in desc.instances], dtype=np.uint32)
    t = np.stack([np.asarray(x, dtype=np.float32) for _, x, _ in desc.instances])
    m = np.array([x for _, _, x in desc.instances], dtype=material_ext_dtype)
    lit = m["base"]["emissive_strength"] > 0
    m["base"]["base_color_factor"] = np.where((lit | (m["bsdf"] == BSDF_DIELECTRIC))[:, None],
                                              m["base"]["base_color_factor"], rng.uniform(0.2, 0.8, size=(len(m), 3)))
    for k in range(len(m)):
        if textures and not lit[k]:
            m[k]["base"]["base_color_index"] = textures[k % 2]
            m[k]["base"]["metallic_roughness_index"] = textures[2]
    return mesh, t, m


def _view(case, rng):
    w, h = case["width"], case["height"]
    j = rng.uniform(-0.02, 0.02, size=3)
    if case.get("scene") == "instanced":
        return scenes.make_view(np.array((50.0, 55.0, -75.0)) + 50 * j, (50.0, 45.0, 50.0), 55.0, w, h)
    if case.get("scene") == "mixed":
        return scenes.make_view(np.array((0.5, 0.38, -0.55)) + j, (0.48, 0.16, 0.45), 45.0, w, h)
    return scenes.make_view(np.array((0.5, 0.5, -1.2)) + j, (0.5, 0.45, 0.5), 45.0, w, h)


def _unit(g, n):
    d = torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    return d / d.norm(dim=1, keepdim=True)


# --------------------------------------------------------------------- prepare

class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case, s.seed = case, seed
    rng = np.random.default_rng(seed)
    _PREPARE[case["kind"]](s, case, rng)
    return s


def _prepare_frame(s, case, rng):
    r = s.r = Renderer(case["width"], case["height"], tlas_metric=case["metric"], instance_bounds=case["bounds"])
    textures, s.env_texture = [], 0
    if case["textured"]:
        noise = rng.integers(0, 256, size=(3, 512, 512, 4), dtype=np.uint8)
        textures = [r.create_texture(noise[0], fmt=1), r.create_texture(noise[1], fmt=1), r.create_texture(noise[2])]
        s.env_texture = r.create_texture(rng.random((256, 512, 4), dtype=np.float32))
    make = _instanced if case["scene"] == "instanced" else functools.partial(_room_instances, textures=textures)
    s.meshes, s.transforms, s.materials = make(r, case, rng)
    s.view = _view(case, rng)
    s.env = (1.0, 1.0, 1.0) if case["textured"] else (0.3, 0.35, 0.4) if case["scene"] == "instanced" else (0.0,) * 3
    s.options = dict(max_bounces=case["bounces"], spp=case["spp"], frame_seed=s.seed & 0xFFFFFF, nee=int(case["nee"]),
                     rr_start_depth=case["rr"], accumulate=False, view_mode=case["view_mode"])
    # the caller's page-locked image buffer
    s.image = torch.zeros(case["height"], case["width"], 4, dtype=torch.float32).pin_memory()
    _submit(s)


def _submit(s):
    s.r.begin_scene(s.view, s.env, s.env_texture)
    s.r.submit_render_meshes(s.meshes, s.transforms, s.materials)
    s.r.end_scene()


def _pick_inputs(case, rng):
    """(transforms, rays): half of the rays towards an instance, half anywhere."""
    n = case["instances"]
    transforms = _transforms(rng, n).astype(np.float32)
    rays = np.zeros(case["rays"], dtype=ray_dtype)
    o = rng.uniform(-20.0, 120.0, size=(len(rays), 3))
    to = transforms[rng.integers(0, n, size=len(rays)), :3, 3] + rng.uniform(-0.6, 0.6, size=(len(rays), 3))
    d = np.where((np.arange(len(rays)) % 2 == 0)[:, None], to - o, rng.normal(size=(len(rays), 3)))
    rays["origin"], rays["dir"] = o, d / np.linalg.norm(d, axis=1, keepdims=True)
    rays["tmin"], rays["tmax"] = 1e-8, FLT_MAX
    return transforms, rays


def _prepare_pick(s, case, rng):
    transforms, s.rays = _pick_inputs(case, rng)
    s.r = Renderer(64, 64)
    mesh = s.r.create_mesh_from_triangles(_sphere(case["freq"], 11), **BVH)
    n = case["instances"]
    s.r.begin_scene(scenes.make_view((50.0, 55.0, -75.0), (50.0, 45.0, 50.0), 55.0, 64, 64))
    s.r.submit_render_meshes(np.full(n, mesh, dtype=np.uint32), transforms, _materials(rng, n))
    s.r.end_scene()


def _prepare_trace(s, case, rng):
    s.r = Renderer(8, 8, blas_layout=case["layout"])
    mesh = s.r.create_mesh_from_triangles(_soup(case["triangles"]), **BVH)
    s.r.begin_scene(scenes.make_view((0.5, 0.5, -0.5), (0.5, 0.5, 0.5), 90.0, 8, 8))
    s.r.submit_render_mesh(mesh, np.eye(4))
    s.r.end_scene()
    g = torch.Generator(device="cuda").manual_seed(s.seed)
    n = case["rays"]
    s.rays = torch.empty(n, 8, device="cuda")
    if case["coherent"]:
        # a pinhole camera's rays in row order, 90 degrees, somewhere before the soup
        side = math.isqrt(n - 1) + 1
        i = torch.arange(n, device="cuda")
        u = ((i % side) + 0.5) / side * 2.0 - 1.0
        v = 1.0 - (torch.div(i, side, rounding_mode="floor") + 0.5) / side * 2.0
        d = torch.stack([u, v, torch.ones_like(u)], dim=1)
        s.rays[:, 0:3] = torch.tensor([0.5, 0.5, -0.5], device="cuda") + 0.1 * (torch.rand(3, generator=g, device="cuda") - 0.5)
        s.rays[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    else:
        s.rays[:, 0:3] = torch.rand(n, 3, generator=g, device="cuda")
        s.rays[:, 4:7] = _unit(g, n)
    s.rays[:, 3] = 1e-8
    s.rays[:, 7] = torch.rand(n, generator=g, device="cuda") if case["any_hit"] else FLT_MAX
    s.hits = torch.zeros(n, 5, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()   # the rays are ready before another stream reads them


def _prepare_blas(s, case, rng):
    s.r = Renderer(8, 8)
    # the mesh as an edit left it: every seed moves the sphere's vertices
    t = _sphere(case["freq"], 11).copy()
    k = rng.uniform(0.9, 1.1, size=3).astype(np.float32)
    for v in ("v0", "v1", "v2"):
        t[v]["position"] *= k
    s.tris = t


def _prepare_tlas(s, case, rng):
    s.r = Renderer(8, 8, tlas_metric=case["metric"])
    n = case["instances"]
    inst = np.zeros(n, dtype=bvh_instance_dtype)
    t = _transforms(rng, n)
    inv = np.linalg.inv(t)
    inst["world_to_local"] = np.transpose(inv, (0, 2, 1)).reshape(n, 16)
    half = np.abs(t[:, :3, :3]).sum(axis=2) * 1.1   # the world box of a displaced unit sphere's box
    inst["aabb_min"], inst["aabb_max"] = t[:, :3, 3] - half, t[:, :3, 3] + half
    inst["bvh_index"] = np.arange(n) % 8
    s.instances = inst


def _prepare_adjoint(s, case, rng):
    r = s.r = Renderer(case["width"], case["height"])
    desc = _room("box", case["subdivision"])
    ids = [r.create_mesh_from_triangles(t, **BVH) for t in desc.meshes]
    r.begin_scene(_view(case, rng), (0.0, 0.0, 0.0))
    for i, l2w, m in desc.instances:
        r.submit_render_mesh(ids[i], l2w, m)
    r.end_scene()
    r.set_albedo(rng.uniform(0.1, 0.9, size=(r.scene_triangle_count(), 3)).astype(np.float32))
    # dloss/dimage of an L2 loss: of the size of the image's own error
    s.dloss = (rng.normal(size=(case["height"], case["width"], 3)) / (case["width"] * case["height"])).astype(np.float32)
    s.options = dict(max_bounces=case["bounces"], spp=case["spp"], frame_seed=s.seed & 0xFFFFFF, nee=int(case["nee"]),
                     rr_start_depth=case["rr"])


def _prepare_batch(s, case, rng):
    s.r = Renderer(8, 8)
    meshes, descs = _batch(case["scenes"], case["tri_lo"], case["tri_hi"], case["max_side"])
    ids = [s.r.create_mesh_from_triangles(t, **BVH) for t in meshes]
    s.b = Batch(s.r)
    for d in descs:
        s.b.begin_scene(d.width, d.height, d.spp, d.view, d.env)
        for k, (mesh, l2w, m) in enumerate(d.instances):
            if k == 0:   # the scene's object, turned
                l2w = scenes.translate_scale((0.0, 0.0, 0.0), 1.0, _rotations(rng, 1)[0])
            s.b.submit(ids[mesh], l2w, m)
        s.b.end_scene()
    s.count = len(descs)
    s.options = dict(max_bounces=case["bounces"], frame_seed=s.seed & 0xFFFFFF, nee=1, rr_start_depth=3)


_PREPARE = dict(frame=_prepare_frame, pick=_prepare_pick, trace=_prepare_trace, blas=_prepare_blas,
                tlas=_prepare_tlas, adjoint=_prepare_adjoint, batch=_prepare_batch)


# ------------------------------------------------------------------------- run

def run(state):
    return _RUN[state.case["kind"]](state, state.case)


def _run_frame(s, case):
    if case["rebuild"]:
        _submit(s)
    s.r.render(**s.options)
    if case["ldr"]:
        return s.r.read_image_ldr()
    s.r.read_image_async(s.image.numpy())
    return s.image


def _run_pick(s, case):
    h = s.r.trace(s.rays, any_hit=case["any_hit"])
    return dict(instance=h["instance"].astype(np.int32), primitive=h["primitive"].astype(np.int32), t=h["t"],
                bary=h["bary"])


def _run_trace(s, case):
    s.r.trace_device(s.rays.data_ptr(), case["rays"], s.hits.data_ptr(), any_hit=case["any_hit"],
                     reorder=case["reorder"])
    return dict(ids=s.hits[:, :2], t_bary=s.hits.view(torch.float32)[:, 2:])   # the five words of hit_result_t


def _run_blas(s, case):
    return s.r.bvh_build(s.tris, **BVH)


def _run_tlas(s, case):
    return s.r.tlas_build(s.instances)


def _run_adjoint(s, case):
    albedo, emission = s.r.adjoint(s.dloss, **s.options)
    return dict(albedo=albedo, emission=emission)


def _run_batch(s, case):
    s.b.render(**s.options)
    return [s.b.read_image(k) for k in range(s.count)]


_RUN = dict(frame=_run_frame, pick=_run_pick, trace=_run_trace, blas=_run_blas, tlas=_run_tlas,
            adjoint=_run_adjoint, batch=_run_batch)


# ------------------------------------------------------------------------ work

# One ray: a descent through a binary tree of the scene's triangles, two box
# tests of 24 operations per level, and one triangle test of 60; a shaded hit
# about 200.
def _ray_flops(triangles):
    return 48.0 * max(1.0, math.log2(max(2, triangles))) + 60.0


def work(case):
    kind = case["kind"]
    if kind == "pick":
        n, tris = case["rays"], 20 * case["freq"] ** 2
        return dict(bytes=52.0 * n, flops=n * _ray_flops(tris * case["instances"]))
    if kind == "trace":
        n = case["rays"]
        # rays in, hits out, the mesh's triangles and nodes once
        return dict(bytes=52.0 * n + 100.0 * case["triangles"], flops=n * _ray_flops(case["triangles"]))
    if kind == "blas":
        n = 20 * case["freq"] ** 2
        # 36 bytes of positions in; nodes (about 32 per triangle), positions and indices out; per level of
        # the tree every triangle binned on three axes and moved
        return dict(bytes=36.0 * n + 72.0 * n, flops=30.0 * n * math.log2(max(2, n / 4)))
    if kind == "tlas":
        n = case["instances"]
        return dict(bytes=92.0 * n + (92.0 + 64.0) * n, flops=30.0 * n * math.log2(max(2, n)))
    if kind == "adjoint":
        paths, tris = case["width"] * case["height"] * case["spp"], 20 * 4 ** case["subdivision"] + 26
        # the image's gradient and the albedo in, the gradients out; every path forward and replayed
        return dict(bytes=12.0 * case["width"] * case["height"] + 24.0 * tris + 200.0 * tris,
                    flops=2.0 * paths * 2.0 * (_ray_flops(tris) + 200.0))
    if kind == "batch":
        _, descs = _batch(case["scenes"], case["tri_lo"], case["tri_hi"], case["max_side"])
        return dict(bytes=sum(16.0 * d.width * d.height + 200.0 * d.sphere_triangles for d in descs),
                    flops=sum(d.paths * 2.0 * (_ray_flops(d.sphere_triangles) + 200.0) for d in descs))
    pixels = case["width"] * case["height"]
    if case["scene"] == "instanced":
        freqs = [max(2, int(round(f * case["detail"]))) for f in scenes.INSTANCED_FREQS]
        stored = 2 * sum(20 * f * f for f in freqs)
        seen = stored / 8 * max(1, case["instances"])
    else:
        stored = seen = sum(len(t) for t in _room(case["scene"], 5).meshes)
    rays = pixels * case["spp"] * (1.0 if case["view_mode"] else 1.4)   # camera rays and the continuing ones
    return dict(bytes=200.0 * stored + pixels * (4.0 if case["ldr"] else 16.0),
                flops=rays * (_ray_flops(seen) + 200.0))


# ----------------------------------------------------------------------- exact

def exact(case, seed):
    """Closest hits in 64 bits, every ray against every triangle.  The other
    families have no such value: a path's next ray starts at a single-precision
    hit and its random choices compare single-precision numbers, so a 64-bit
    path soon leaves the one that was rendered; an any-hit query returns
    whichever hit its traversal meets first; builders return integers and
    copies of their input."""
    if case["kind"] != "pick" or case["any_hit"] or case["rays"] * case["instances"] * case["freq"] ** 2 > 2e8:
        return None
    transforms, rays = _pick_inputs(case, np.random.default_rng(seed))
    f64 = dict(dtype=torch.float64, device="cuda")
    mesh = _sphere(case["freq"], 11)
    v = [torch.tensor(mesh[k]["position"], **f64) for k in ("v0", "v1", "v2")]
    o = torch.tensor(rays["origin"], **f64)
    d = torch.tensor(rays["dir"], **f64)
    n = len(o)
    best = torch.full((n,), FLT_MAX, **f64)
    u_best, v_best = torch.zeros(n, **f64), torch.zeros(n, **f64)
    for m in transforms:
        w2l = torch.linalg.inv(torch.tensor(m, **f64))
        lo, ld = o @ w2l[:3, :3].T + w2l[:3, 3], d @ w2l[:3, :3].T
        e1, e2 = v[1] - v[0], v[2] - v[0]
        step = max(1, 4_000_000 // len(e1))
        for a in range(0, n, step):
            b = min(n, a + step)
            p = torch.linalg.cross(ld[a:b, None], e2[None])
            det = (e1 * p).sum(-1)
            tv = lo[a:b, None] - v[0]
            q = torch.linalg.cross(tv, e1[None].expand_as(tv))
            u, w = (tv * p).sum(-1) / det, (ld[a:b, None] * q).sum(-1) / det
            t = (e2 * q).sum(-1) / det
            hit = (det >= 1e-8) & (u >= 0) & (w >= 0) & (u + w <= 1) & (t >= 0)
            t = torch.where(hit, t, torch.inf)
            tb, k = t.min(dim=1)
            row = torch.arange(b - a, device="cuda")
            near = tb < best[a:b]
            best[a:b] = torch.where(near, tb, best[a:b])
            u_best[a:b] = torch.where(near, u[row, k], u_best[a:b])
            v_best[a:b] = torch.where(near, w[row, k], v_best[a:b])
    return dict(instance=None, primitive=None, t=best.cpu().numpy(),
                bary=torch.stack([u_best, v_best], dim=1).cpu().numpy())
