"""The work that a user of pike_gb300 has it do, as measurable cases.

Every case goes through the package's public entry points (the C ABI bound by
``Context``, ``PikeRenderer``, ``Batch`` and ``diff.render``) and returns what
the call computes, whole.  The kinds:

``query``   rays in device buffers against a loaded scene (pk_cast_rays):
            picking, visibility and baking, from a few hundred rays up.
``frames``  progressive rendering: a number of samples per pixel of one view
            (pk_render_frames), then the mean image and the 8-bit display.
``viewer``  one PikeRenderer.tick() and its image: an interactive viewer that
            shows every sample, through one call per tick or pass by pass.
``batch``   many requests of uneven size over resident scenes (Batch).
``train``   one inverse-rendering step: differentiable render, L2 loss,
            gradients of albedo, roughness and environment (diff.render).
``build``   the BVH of a scene whose geometry changed (pk_bvh_build), with
            the compressed 8-wide tree beside it where the context traces it.
``env``     the sampling tables of a new environment map (pk_env_build).

Scenes are seeded and of the shapes the benchmark and the tests use: a ground
quad with boxes, a displaced icosphere in an open box with 256 material
groups, a triangle soup, and log-normal environments with a sun.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from pike_gb300 import _lib, diff, synth
from pike_gb300._lib import Context, camera_struct, ptr
from pike_gb300.batch import Batch, Request, orbit_camera, scene_context
from pike_gb300.passes import GPUDevice
from pike_gb300.renderer import PikeRenderer
from pike_gb300.scene import Scene

MISS_T = 100000.0  # the distance of a ray that hits nothing
BRUTE_FORCE = 2e9  # ray-triangle pairs that exact() still tests one by one


def listed():
    return [
        # a mouse pick or a few probes in an editor: latency is all there is
        dict(name="query_pick", kind="query", scene="boxes", detail=64, rays=257, any_hit=False, noalloc=True,
             coherent=True),
        # visibility of a million point pairs (light baking) in a mid-sized mesh
        dict(name="query_visibility", kind="query", scene="sphere", detail=7, rays=999_983, any_hit=True,
             noalloc=False, coherent=False),
        # incoherent closest hits in the 1.3M-triangle mesh: ambient occlusion and probe baking
        dict(name="query_closest", kind="query", scene="sphere", detail=8, rays=2_097_143, any_hit=False,
             noalloc=False, coherent=False),
        # the small scene's preview: 256x256, 4 samples per pixel, 4 bounces
        dict(name="frames_preview", kind="frames", scene="boxes", detail=64, width=256, height=256, spp=4, bounces=4,
             in_flight=4, trace="persistent", kahan=False, alias=False),
        # the headline: the 1.3M-triangle scene at 1080p, 8 bounces, frames in flight
        dict(name="frames_1080p", kind="frames", scene="sphere", detail=8, width=1920, height=1080, spp=8, bounces=8,
             in_flight=8, trace="persistent", kahan=False, alias=False),
        # the precision form on a soup: 8-wide tree, compensated sums, alias-table light sampling
        dict(name="frames_wide_soup", kind="frames", scene="soup", detail=524_288, width=1280, height=720, spp=4,
             bounces=4, in_flight=4, trace="wide", kahan=True, alias=True),
        # an interactive viewer at an odd window size, one call per tick
        dict(name="viewer_tick", kind="viewer", scene="sphere", detail=6, width=853, height=479, bounces=4, fused=True,
             batch_size=853 * 479),
        # the pass API driven pass by pass, in batches that do not divide the image
        dict(name="viewer_passes", kind="viewer", scene="boxes", detail=833, width=640, height=360, bounces=4,
             fused=False, batch_size=100_000),
        # thumbnails and previews of three scenes at uneven sizes in one launch
        dict(name="batch_requests", kind="batch", requests=16, most=1280, spp=16, detail=7),
        # one step of inverse rendering at the differentiation workload's size
        dict(name="train_step", kind="train", detail=8, width=512, height=512, spp=16, depth=4, env=256),
        # a deformed 1.3M-triangle mesh: its BVH is rebuilt
        dict(name="build_large", kind="build", scene="sphere", detail=8, wide=False),
        # a new 2048x1024 environment map is loaded
        dict(name="env_large", kind="env", width=2048, height=1024, alias=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query", "query", "frames", "frames", "viewer", "batch", "train", "build", "build", "env"])
    scene, detail = rng.choice([("boxes", rng.choice([16, 64, 833])), ("sphere", rng.randint(4, 8)),
                                ("sphere", rng.randint(5, 8)), ("soup", _log_int(rng, 2000, 524_288))])
    if kind == "query":
        noalloc = rng.random() < 0.3
        return dict(kind=kind, scene=scene, detail=detail, rays=_log_int(rng, 100, 1 << 20 if noalloc else 1 << 21),
                    any_hit=rng.random() < 0.5, noalloc=noalloc, coherent=rng.random() < 0.4)
    if kind == "frames":
        h = _log_int(rng, 90, 1080)
        return dict(kind=kind, scene=scene, detail=detail, width=max(64, int(h * rng.uniform(1.0, 1.78))), height=h,
                    spp=rng.choice([1, 2, 4, 8]), bounces=rng.randint(2, 8), in_flight=rng.choice([1, 4, 4, 8]),
                    trace=rng.choice(["persistent", "persistent", "wide"]), kahan=rng.random() < 0.25,
                    alias=rng.random() < 0.25)
    if kind == "viewer":
        h = _log_int(rng, 90, 720)
        w = max(64, int(h * rng.uniform(1.0, 1.78)))
        return dict(kind=kind, scene=scene, detail=detail, width=w, height=h, bounces=rng.randint(2, 6),
                    fused=rng.random() < 0.6, batch_size=rng.choice([w * h, w * h, w * h // 2 + 77]))
    if kind == "batch":
        return dict(kind=kind, requests=rng.randint(2, 16), most=_log_int(rng, 160, 1280), spp=rng.choice([1, 4, 16]),
                    detail=rng.randint(5, 7))
    if kind == "train":
        h = _log_int(rng, 32, 512)
        return dict(kind=kind, detail=rng.randint(4, 8), width=min(512, max(32, int(h * rng.uniform(1.0, 1.5)))),
                    height=h, spp=rng.choice([1, 4, 16]), depth=rng.randint(2, 4), env=rng.choice([32, 64, 128, 256]))
    if kind == "build":
        return dict(kind=kind, scene=scene, detail=detail, wide=rng.random() < 0.4)
    w = _log_int(rng, 64, 2048)
    return dict(kind=kind, width=w, height=max(16, w // 2 + rng.choice([0, 0, 1])), alias=rng.random() < 0.4)


# ---------------------------------------------------------------- scenes
@functools.lru_cache(maxsize=None)
def _icosphere(subdivisions):
    return synth.icosphere(subdivisions)


def _normals(pos, faces):
    a, b, c = pos[faces[:, 0]], pos[faces[:, 1]], pos[faces[:, 2]]
    fn = np.cross(b - a, c - a)
    n = np.stack([sum(np.bincount(faces[:, k], fn[:, x], pos.shape[0]) for k in range(3)) for x in range(3)], 1)
    return n / np.sqrt((n * n).sum(1))[:, None]


def _tangents(n):
    up = np.where(np.abs(n[:, 1:2]) < 0.999, np.array([[0.0, 1.0, 0.0]]), np.array([[1.0, 0.0, 0.0]]))
    t = np.cross(n, up)
    return np.concatenate([t / np.sqrt((t * t).sum(1))[:, None], np.ones((n.shape[0], 1))], 1)


def _radiance(width, height, rng, sigma=1.5, sun=1e4):
    """Log-normal grey texels and a 4x4-texel sun at a random place."""
    L = np.exp(sigma * rng.standard_normal((height, width)))
    y, x = int(rng.integers(0, height - 4)), int(rng.integers(0, width - 4))
    L[y:y + 4, x:x + 4] = sun
    return np.repeat(L[..., None], 3, axis=2).astype(np.float32)


def _source(pos, normal, tangent, tris, materials, env):
    return synth.SceneSource(name="case", pos=pos, normal=normal, tangent=tangent, uv=np.full((pos.shape[0], 2), 0.5),
                             tris=np.ascontiguousarray(tris, np.int32), materials=materials, env_rgbe=env,
                             env_hdr=None, cam_pos=(0, 0, -1), cam_target=(0, 0, 0), fov=math.pi / 3, width=64,
                             height=64, spp=1, bounces=4)


def _sphere(subdivisions, rng, env):
    """A displaced icosphere of radius 1.5 with 256 material groups in an open 10x10x10 box."""
    v, f = _icosphere(subdivisions)
    k = rng.normal(size=(6, 3)) * 5.0
    wave = sum(np.sin(v @ k[i] + rng.uniform(0, 6.28)) for i in range(6)) / 6.0
    pos = v * (1.5 * (1.0 + 0.1 * wave))[:, None]
    nrm = _normals(pos, f)
    groups = 256
    mats = np.zeros((groups + 1, 9))
    mats[:, 0:3] = rng.uniform(0.1, 0.9, (groups + 1, 3))
    mats[:, 3] = 1.0
    mats[:, 4] = rng.uniform(0.05, 1.0, groups + 1)
    mats[:, 5] = rng.random(groups + 1) < 0.5
    mats[groups] = [0.7, 0.7, 0.7, 1.0, 1.0, 0.0, 0.0, 0.0, 0.0]
    tris = [np.concatenate([f, ((np.arange(f.shape[0]) * groups) // f.shape[0])[:, None]], 1)]
    P, N, T = [pos], [nrm], [_tangents(nrm)]
    base = pos.shape[0]
    for axis, sign in ((0, 1), (0, -1), (1, -1), (2, 1), (2, -1)):  # open towards +y
        a, b = (axis + 1) % 3, (axis + 2) % 3
        q = np.zeros((4, 3))
        q[:, axis] = 5.0 * sign
        q[:, a] = [-5, 5, 5, -5]
        q[:, b] = [-5, -5, 5, 5]
        n, t = np.zeros((4, 3)), np.zeros((4, 4))
        n[:, axis], t[:, a], t[:, 3] = -sign, 1.0, 1.0
        P.append(q)
        N.append(n)
        T.append(t)
        tris.append(np.array([[base, base + 1, base + 2, groups], [base, base + 2, base + 3, groups]]))
        base += 4
    return _source(np.concatenate(P), np.concatenate(N), np.concatenate(T), np.concatenate(tris), mats, env)


def _soup(n, rng, env):
    """Triangles with centroids uniform in a 100^3 cube and sizes log-uniform in [0.01, 1]."""
    c = rng.uniform(-50.0, 50.0, (n, 3))
    size = np.exp(rng.uniform(math.log(0.01), 0.0, (n, 1)))
    a, b = (rng.normal(size=(n, 3)) for _ in range(2))
    a, b = (x / np.sqrt((x * x).sum(1))[:, None] * size for x in (a, b))
    pos = np.stack([c + a, c + b, c - a - b], 1).reshape(-1, 3)
    fn = np.cross(b - a, -2.0 * a - b)
    nrm = np.repeat(fn / np.maximum(np.sqrt((fn * fn).sum(1)), 1e-30)[:, None], 3, axis=0)
    tris = np.concatenate([np.arange(3 * n).reshape(n, 3), np.zeros((n, 1), np.int64)], 1)
    return _source(pos, nrm, _tangents(nrm), tris, np.array([[0.6, 0.6, 0.6, 1.0, 0.5, 0.0, 0.0, 0.0, 0.0]]), env)


def _scene(kind, detail, seed):
    rng = np.random.default_rng(seed)
    if kind == "boxes":
        return synth.small_scene(seed_index=seed, n_boxes=detail)
    big = kind == "sphere" and detail >= 8
    env = synth.rgbe_encode(_radiance(2048 if big else 512, 1024 if big else 256, rng))
    return _sphere(detail, rng, env) if kind == "sphere" else _soup(detail, rng, env)


def _triangles(kind, detail):
    return {"boxes": 2 + 12 * detail, "sphere": 20 * 4 ** detail + 10 if detail < 16 else 0, "soup": detail}[kind]


def _frame(pos):
    """The normalised frame the passes work in: centre and scale of the scene's box."""
    lo, hi = pos.min(0), pos.max(0)
    span = hi - lo
    return lo + span * 0.5, 2.0 / max(span[0], span[1], span[2])


def _camera(kind, src, seed):
    """A pinhole camera on a circle around the scene, looking at its middle."""
    angle = float(np.random.default_rng([seed, 1]).uniform(0.0, 2.0 * math.pi))
    radius, height = {"boxes": (20.0, 8.0), "sphere": (4.5, 1.5), "soup": (120.0, 10.0)}[kind]
    eye = np.array([radius * math.sin(angle), height, -radius * math.cos(angle)])
    centre, scale = _frame(src.pos)
    d = -eye / math.sqrt(float(eye @ eye))
    return dict(pos=[float(np.float32(v)) for v in (eye - centre) * scale], dir=[float(np.float32(v)) for v in d],
                fov=float(np.float32(math.pi / 3)), focalDepth=0.5, apertureSize=0.0, distortion=0.0, bokeh=0.5,
                invocationOffset=0)


def _load(ctx, src):
    tr = np.zeros(3)
    ctx.call("pk_scene_flatten", ptr(np.ascontiguousarray(src.pos)), ptr(np.ascontiguousarray(src.normal)),
             ptr(np.ascontiguousarray(src.tangent)), ptr(np.ascontiguousarray(src.uv)), src.pos.shape[0],
             ptr(src.tris), src.tris.shape[0], 1.0, ptr(tr))
    ctx.call("pk_materials_set", ptr(src.materials), src.materials.shape[0])


# ---------------------------------------------------------------- the kinds
def _rays(case, src, seed):
    """Origins and directions: a view's pixel rays, or points in the scene looking anywhere."""
    n = case["rays"]
    rng = np.random.default_rng([seed, 2])
    o, d = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    if case["coherent"]:
        cam = _camera(case["scene"], src, seed)
        f = np.array(cam["dir"])
        x = np.cross(f, [0.0, 1.0, 0.0])
        x /= np.sqrt(x @ x)
        y = np.cross(x, f)
        w = max(1, int(math.sqrt(n)))
        i = np.arange(n)
        u = ((i % w) + rng.random(n)) / w * 2.0 - 1.0
        v = ((i // w) + rng.random(n)) / (n // w + 1) * 2.0 - 1.0
        dirs = f + 0.577 * (u[:, None] * x + v[:, None] * y)
        o[:, :3] = cam["pos"]
    else:
        dirs = rng.normal(size=(n, 3))
        o[:, :3] = rng.uniform(-0.9, 0.9, (n, 3))
    d[:, :3] = dirs / np.sqrt((dirs * dirs).sum(1))[:, None]
    return o, d


def _prepare_query(case, seed):
    src = _scene(case["scene"], case["detail"], seed)
    ctx = Context(0)
    ctx.call("pk_configure", 64, 64, 64 * 64)
    _load(ctx, src)
    ctx.call("pk_bvh_build", _lib.PK_BVH_SWEEP)
    o, d = _rays(case, src, seed)
    n = case["rays"]
    hits = torch.zeros((n, 4), dtype=torch.int32, device="cuda")
    return dict(ctx=ctx, o=torch.from_numpy(o).cuda(), d=torch.from_numpy(d).cuda(), hits=hits,
                index=torch.zeros(n, dtype=torch.int32, device="cuda"),
                count=torch.zeros(1, dtype=torch.int32, device="cuda"),
                call="pk_cast_rays_noalloc" if case["noalloc"] else "pk_cast_rays", any_hit=int(case["any_hit"]))


def _run_query(s):
    s["ctx"].call(s["call"], s["o"].data_ptr(), s["d"].data_ptr(), s["o"].shape[0], s["any_hit"],
                  s["hits"].data_ptr(), s["index"].data_ptr(), s["count"].data_ptr())
    h = s["hits"]
    return dict(t=h.view(torch.float32)[:, 0], triangle=h[:, 1], bary=h[:, 2], index=s["index"], count=s["count"])


def _prepare_frames(case, seed):
    src = _scene(case["scene"], case["detail"], seed)
    w, h = case["width"], case["height"]
    ctx = Context(0)
    ctx.call("pk_configure", w, h, w * h)
    _load(ctx, src)
    ctx.call("pk_bvh_build", _lib.PK_BVH_SWEEP)
    ctx.call("pk_env_build", ptr(src.env_rgbe), src.env_rgbe.shape[1], src.env_rgbe.shape[0])
    ctx.call("pk_set_trace_mode", _lib.PK_TRACE_PERSISTENT | (_lib.PK_TRACE_WIDE if case["trace"] == "wide" else 0))
    ctx.call("pk_set_accumulation", _lib.PK_ACCUM_COMPENSATED if case["kahan"] else _lib.PK_ACCUM_RUNNING_MEAN)
    ctx.call("pk_set_env_sampling", _lib.PK_ENV_ALIAS if case["alias"] else _lib.PK_ENV_HISTOGRAM)
    ctx.call("pk_set_frames_in_flight", case["in_flight"])
    ctx.call("pk_set_camera", camera_struct(_camera(case["scene"], src, seed)))
    return dict(ctx=ctx, spp=case["spp"], bounces=case["bounces"], theta=float(seed % 7),
                mean=ctx.pinned((h, w, 4), np.float32), shown=ctx.pinned((h, w, 4), np.uint8))


def _run_frames(s):
    ctx = s["ctx"]
    ctx.call("pk_set_render_state", 0, s["theta"])
    ctx.call("pk_render_frames", s["spp"], s["bounces"])
    ctx.call("pk_read_accum", ptr(s["mean"].array))
    ctx.call("pk_read_display", None, ptr(s["shown"].array))
    ctx.call("pk_sync")
    return dict(mean=s["mean"].array, shown=s["shown"].array)


def _prepare_viewer(case, seed):
    src = _scene(case["scene"], case["detail"], seed)
    r = PikeRenderer(Scene.from_source(src), (case["width"], case["height"]), _camera(case["scene"], src, seed),
                     device=GPUDevice(0), num_bounces=case["bounces"], batch_size=case["batch_size"],
                     fused=case["fused"])
    r.initWebGpu()
    r.device.ctx.call("pk_set_frames_in_flight", 1)  # every sample is shown before the next
    r.renderState.setEnvRotation(float(seed % 7))
    ctx = r.device.ctx
    shape = (case["height"], case["width"], 4)
    return dict(r=r, mean=ctx.pinned(shape, np.float32), shown=ctx.pinned(shape, np.uint8))


def _run_viewer(s):
    r = s["r"]
    r.renderState.resetSamples()
    r.tick()
    ctx = r.device.ctx
    ctx.call("pk_read_accum", ptr(s["mean"].array))
    ctx.call("pk_read_display", None, ptr(s["shown"].array))
    return dict(mean=s["mean"].array, shown=s["shown"].array)


def _requests(case, seed):
    """Resolutions log-uniform from 128 pixels wide up, samples a power of four, depth 4 to 8."""
    rng = np.random.default_rng([case["requests"], case["most"], case["spp"], case["detail"]])  # the load: the case's
    cams = np.random.default_rng([seed, 3])  # the views: the seed's
    out = []
    for i in range(case["requests"]):
        w = int(round(128 * (max(case["most"], 128) / 128) ** (1.0 if i == 0 else rng.uniform())))
        out.append(Request(scene=i % 3, width=w, height=max(64, int(w * 0.5625) | 1),
                           spp=int(rng.choice([x for x in (1, 4, 16) if x <= case["spp"]])),
                           depth=int(rng.integers(4, 9)), camera=orbit_camera(cams)))
    return sorted(out, key=lambda q: q.paths)


def _prepare_batch(case, seed):
    scenes = [_scene("boxes", 833, seed), _scene("sphere", case["detail"] - 1, seed),
              _scene("sphere", case["detail"], seed + 1)]
    b = Batch([scene_context(s) for s in scenes])
    b.set_requests(_requests(case, seed))
    return b


def _run_batch(b):
    b.reset()
    b.render(1)
    return [b.image(i) for i in range(len(b.requests))]


def _prepare_train(case, seed):
    src = _scene("sphere", case["detail"], seed)
    scene = diff.DiffScene(src, case["width"], case["height"], spp=case["spp"], depth=case["depth"],
                           camera=_camera("sphere", src, seed))
    rng = np.random.default_rng([seed, 4])
    dev = dict(dtype=torch.float32, device="cuda")
    env = torch.tensor(_radiance(case["env"], case["env"] // 2, rng, sigma=1.0, sun=20.0), **dev)
    m = src.materials
    return dict(scene=scene, seed=int(seed) % 1000, env=env.requires_grad_(True),
                albedo=torch.tensor(m[:, 0:3], **dev).requires_grad_(True),
                rough=torch.tensor(m[:, 4], **dev).requires_grad_(True),
                target=torch.tensor(rng.random((case["height"], case["width"], 4)), **dev))


def _run_train(s):
    p = [s["albedo"], s["rough"], s["env"]]
    for x in p:
        x.grad = None
    image = diff.render(s["scene"], *p, seed=s["seed"], grad_seed=s["seed"] + 1)
    loss = diff.l2_loss(image, s["target"])
    loss.backward()
    return dict(image=image.detach(), loss=loss.detach(), albedo=p[0].grad, rough=p[1].grad, env=p[2].grad)


def _zeroed(ctx, shape, dtype):
    """Page-locked memory that a download fills from its start, as far as this input goes."""
    a = ctx.pinned(shape, dtype)
    a.array[...] = 0
    return a


def _prepare_build(case, seed):
    src = _scene(case["scene"], case["detail"], seed)
    ctx = Context(0)
    ctx.call("pk_configure", 64, 64, 64 * 64)
    _load(ctx, src)
    t = src.tris.shape[0]
    if case["wide"]:  # a context that traces the 8-wide tree keeps it beside every BVH it builds
        ctx.call("pk_bvh_build", _lib.PK_BVH_SWEEP)
        ctx.call("pk_set_trace_mode", _lib.PK_TRACE_PERSISTENT | _lib.PK_TRACE_WIDE)
    s = dict(ctx=ctx, wide=case["wide"], nodes=_zeroed(ctx, (2 * t, 5), np.int32), tris=_zeroed(ctx, (t, 4), np.int32),
             verts=_zeroed(ctx, (src.pos.shape[0], 4), np.float32))
    if case["wide"]:
        s.update(wnodes=_zeroed(ctx, (t + 8, 20), np.int32), wtris=_zeroed(ctx, (t, 12), np.int32))
    return s


def _run_build(s):
    ctx = s["ctx"]
    ctx.call("pk_bvh_build", _lib.PK_BVH_SWEEP)
    nodes, leaves = C.c_uint32(), C.c_uint32()
    norm = np.zeros(4)
    ctx.call("pk_bvh_info", C.byref(nodes), C.byref(leaves), ptr(norm))
    ctx.call("pk_bvh_download", ptr(s["nodes"].array), ptr(s["tris"].array), ptr(s["verts"].array))
    out = dict(count=[nodes.value, leaves.value], nodes=s["nodes"].array, tris=s["tris"].array, verts=s["verts"].array,
               norm=norm)
    if s["wide"]:
        n, depth = C.c_uint32(), C.c_uint32()
        ctx.call("pk_wide_info", C.byref(n), C.byref(depth))
        ctx.call("pk_wide_download", ptr(s["wnodes"].array), ptr(s["wtris"].array))
        out.update(wide_count=[n.value, depth.value], wide_nodes=s["wnodes"].array, wide_tris=s["wtris"].array)
    return out


def _env_image(case, seed):
    return synth.rgbe_encode(_radiance(case["width"], case["height"], np.random.default_rng([seed, 5])))


def _prepare_env(case, seed):
    ctx = Context(0)
    ctx.call("pk_configure", 64, 64, 64 * 64)
    image = np.ascontiguousarray(_env_image(case, seed))
    h, w = image.shape[:2]
    s = dict(ctx=ctx, image=image, alias=case["alias"], bins=_zeroed(ctx, (1024, 2), np.int32),
             coords=_zeroed(ctx, (h * w, 2), np.int32), pdf=_zeroed(ctx, (h, w), np.float32))
    if case["alias"]:  # a context that samples by the alias table keeps it beside every map it loads
        ctx.call("pk_env_build", ptr(image), w, h)
        ctx.call("pk_set_env_sampling", _lib.PK_ENV_ALIAS)
        s.update(table=_zeroed(ctx, (h * w, 2), np.int32), alias_pdf=_zeroed(ctx, (h, w), np.float32))
    return s


def _run_env(s):
    ctx, (h, w) = s["ctx"], s["image"].shape[:2]
    ctx.call("pk_env_build", ptr(s["image"]), w, h)
    nb = C.c_uint32()
    ctx.call("pk_env_info", None, None, C.byref(nb))
    ctx.call("pk_env_download", ptr(s["bins"].array), ptr(s["coords"].array), ptr(s["pdf"].array))
    out = dict(count=nb.value, bins=s["bins"].array, coords=s["coords"].array, pdf=s["pdf"].array)
    if s["alias"]:
        ctx.call("pk_env_alias_download", ptr(s["table"].array), ptr(s["alias_pdf"].array))
        out.update(table=s["table"].array, alias_pdf=s["alias_pdf"].array)
    return out


_PREPARE = dict(query=_prepare_query, frames=_prepare_frames, viewer=_prepare_viewer, batch=_prepare_batch,
                train=_prepare_train, build=_prepare_build, env=_prepare_env)
_RUN = dict(query=_run_query, frames=_run_frames, viewer=_run_viewer, batch=_run_batch, train=_run_train,
            build=_run_build, env=_run_env)


def prepare(case, seed):
    return case["kind"], _PREPARE[case["kind"]](case, seed)


def run(state):
    kind, s = state
    return _RUN[kind](s)


# ---------------------------------------------------------------- work
def _ray_flops(tris):
    """One descent of a binary tree (two slab tests a level) and two triangle tests."""
    return 48.0 * max(1.0, math.log2(tris)) + 2 * 60.0


SHADE_FLOPS = 600.0  # interpolation, GGX sampling and evaluation, light sampling, two pdfs


def work(case):
    kind = case["kind"]
    if kind == "query":
        n = case["rays"]
        return dict(bytes=n * (32.0 + 16.0 + 4.0), flops=n * _ray_flops(_triangles(case["scene"], case["detail"])))
    if kind in ("frames", "viewer"):
        # about two camera-path rays and as many shadow rays a sample survive at least; the scene is read
        # once and the image written once
        tris = _triangles(case["scene"], case["detail"])
        px = case["width"] * case["height"]
        paths = px * case.get("spp", 1)
        return dict(bytes=px * 20.0 + tris * (48.0 + 16.0 + 20.0),
                    flops=paths * 2.0 * (2.0 * _ray_flops(tris) + SHADE_FLOPS))
    if kind == "batch":
        reqs = _requests(case, 0)
        tris = [2 + 12 * 833, _triangles("sphere", case["detail"] - 1), _triangles("sphere", case["detail"])]
        return dict(bytes=sum(16.0 * q.width * q.height for q in reqs) + sum(84.0 * t for t in tris),
                    flops=sum(q.paths * 2.0 * (2.0 * _ray_flops(tris[q.scene]) + SHADE_FLOPS) for q in reqs))
    if kind == "train":
        tris = _triangles("sphere", case["detail"])
        paths = case["width"] * case["height"] * case["spp"]
        px, texels = case["width"] * case["height"], case["env"] * case["env"] // 2
        return dict(bytes=px * 16.0 * 4 + texels * 12.0 * 3 + tris * 84.0,
                    flops=paths * 2.0 * 2.0 * (2.0 * _ray_flops(tris) + SHADE_FLOPS))  # a render and its replay
    if kind == "build":
        # positions and indices in; nodes (about one per triangle at the least), triangles and vertices out
        tris = _triangles(case["scene"], case["detail"])
        verts = 3 * tris if case["scene"] == "soup" else tris // 2 + 2 if case["scene"] == "sphere" else 2 * tris
        return dict(bytes=verts * (24.0 + 16.0) + tris * (16.0 + 20.0 + 16.0) + (tris * 68.0 if case["wide"] else 0.0),
                    flops=tris * 30.0 * max(1.0, math.log2(tris)))
    n = case["width"] * case["height"]
    return dict(bytes=n * (4.0 + 8.0 + 4.0 + (12.0 if case["alias"] else 0.0)), flops=n * 20.0)


# ---------------------------------------------------------------- 64 bits
def _exact_query(case, seed):
    """Closest distances by Moeller-Trumbore over every triangle."""
    if case["any_hit"] or case["rays"] * _triangles(case["scene"], case["detail"]) > BRUTE_FORCE:
        return None
    src = _scene(case["scene"], case["detail"], seed)
    centre, scale = _frame(src.pos)
    o, d = (torch.from_numpy(x[:, :3].astype(np.float64)).cuda() for x in _rays(case, src, seed))
    v = torch.from_numpy((src.pos - centre) * scale).cuda()
    f = torch.from_numpy(src.tris[:, :3].astype(np.int64)).cuda()
    a, e1, e2 = v[f[:, 0]], v[f[:, 1]] - v[f[:, 0]], v[f[:, 2]] - v[f[:, 0]]
    best = torch.full((o.shape[0],), MISS_T, dtype=torch.float64, device="cuda")
    step = max(1, int(2e7 / a.shape[0]))
    for i in range(0, o.shape[0], step):
        oo, dd = o[i:i + step, None, :], d[i:i + step, None, :]
        p = torch.linalg.cross(dd.expand(-1, a.shape[0], -1), e2[None].expand(dd.shape[0], -1, -1))
        det = (e1 * p).sum(-1)
        w = oo - a
        q = torch.linalg.cross(w, e1[None].expand_as(w))
        u, vv, t = (w * p).sum(-1) / det, (dd * q).sum(-1) / det, (e2 * q).sum(-1) / det
        ok = (det.abs() >= 1e-8) & (u >= 0) & (u <= 1) & (vv >= 0) & (u + vv <= 1) & (t > 1e-8)
        best[i:i + step] = torch.where(ok, t, torch.full_like(t, MISS_T)).min(1).values
    return dict(t=best, triangle=None, bary=None, index=None, count=None)


def _exact_build(case, seed):
    src = _scene(case["scene"], case["detail"], seed)
    centre, scale = _frame(src.pos)
    verts = np.zeros((src.pos.shape[0], 4))
    verts[:, :3] = (src.pos - centre) * scale
    out = dict(count=None, nodes=None, tris=None, verts=verts, norm=np.concatenate([centre, [scale]]))
    if case["wide"]:
        out.update(wide_count=None, wide_nodes=None, wide_tris=None)
    return out


def _exact_env(case, seed):
    """The pdf of the equal-mass luminance histogram."""
    c = _env_image(case, seed).reshape(-1, 4).astype(np.float64)
    rad = np.ldexp(0.2126 * c[:, 0] + 0.7152 * c[:, 1] + 0.0722 * c[:, 2], c[:, 3].astype(np.int64) - 128) / 255.0
    order = np.argsort(-rad, kind="stable")
    r = rad[order]
    total = np.cumsum(rad)[-1]
    size = total / min(256.0, max(32.0, 2.0 * math.ceil(total / rad.max())))
    edges = [0]
    while True:  # a bin ends where its running sum reaches the size
        ahead, end = 1024, None
        while end is None:
            s = np.cumsum(r[edges[-1]:edges[-1] + ahead])
            k = int(np.searchsorted(s, size))
            if k < s.size:
                end = edges[-1] + k + 1
            elif edges[-1] + ahead >= r.size:
                end = r.size
            ahead *= 4
        if end >= r.size:
            break
        edges.append(end)
    edges.append(r.size)
    count = np.diff(edges)
    pdf = np.empty(r.size)
    pdf[order] = np.repeat((1.0 / count.size) * (r.size / count) / (2.0 * math.pi ** 2), count)
    pdf = pdf.reshape(case["height"], case["width"])
    out = dict(count=None, bins=None, coords=None, pdf=pdf)
    if case["alias"]:
        out.update(table=None, alias_pdf=rad.reshape(pdf.shape) / total * r.size / (2.0 * math.pi ** 2))
    return out


def exact(case, seed):
    """Distances, vertices and pdfs; a path tracer's images have no value without its own random numbers."""
    f = dict(query=_exact_query, build=_exact_build, env=_exact_env).get(case["kind"])
    return None if f is None else f(case, seed)
