"""The builders and wavefront kernels at the sizes where their tiles, blocks and
dispatch rules change, bit for bit against the oracle (or against the same work
cut differently, where the oracle would take too long)."""
import ctypes as C

import numpy as np
import pytest

from pike_gb300 import _lib, synth
from pike_gb300._lib import Context, ptr

from helpers import Pair, assert_bits_equal, assert_bits_equal_nan, camera_struct

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(pk_built):
    return Context(0)


def soup(n, seed, spread=1.0, offset=0.0):
    rng = np.random.default_rng(seed)
    c = rng.uniform(-spread, spread, (n, 1, 3)) + offset
    pos = (c + rng.normal(size=(n, 3, 3)) * 0.02 * spread).reshape(-1, 3)
    tris = np.concatenate([np.arange(3 * n).reshape(n, 3), np.zeros((n, 1), np.int64)], 1).astype(np.int32)
    return pos, tris


def quads(n):
    """An n x n grid of axis-aligned quads: every box and many costs tie exactly."""
    x, y = (a.reshape(-1) for a in np.meshgrid(np.arange(n, dtype=float), np.arange(n, dtype=float)))
    corner = np.array([[0, 0], [1, 0], [1, 1], [0, 1]], float)
    pos = np.zeros((n * n, 4, 3))
    pos[..., 0] = x[:, None] + corner[:, 0]
    pos[..., 2] = y[:, None] + corner[:, 1]
    base = 4 * np.arange(n * n)[:, None, None]
    t = (base + np.array([[0, 1, 2], [0, 2, 3]])[None]).reshape(-1, 3)
    return pos.reshape(-1, 3), np.concatenate([t, np.zeros((t.shape[0], 1), np.int64)], 1).astype(np.int32)


def clusters(n):
    """Dense clusters a million times smaller than the scene: rounded boxes that cannot tell costs apart."""
    pos, tris = soup(n, 5, spread=1e-6)
    rng = np.random.default_rng(6)
    shift = rng.uniform(-1, 1, (4, 3))[rng.integers(0, 4, n)]
    return (pos.reshape(n, 3, 3) + shift[:, None, :]).reshape(-1, 3), tris


BVH_CASES = {**{f"soup{n}": (lambda n=n: soup(n, n)) for n in (1, 2, 33, 511, 512, 513, 1024, 1025, 2049, 5000)},
             "far": lambda: soup(1500, 3, spread=1e-3, offset=1e5), "quads16": lambda: quads(16),
             "quads40": lambda: quads(40), "clusters": lambda: clusters(3000)}


@pytest.mark.parametrize("name", list(BVH_CASES))
def test_sweep_build_matches_oracle(ctx, oracle, name):
    """One block's subtree (up to 512 triangles), tiles of 1024, ties and scales."""
    pos, tris = BVH_CASES[name]()
    pos = np.ascontiguousarray(pos)
    ref = oracle.BVH(pos, tris)
    attrs = np.zeros((pos.shape[0], 4), np.uint32)
    ctx.call("pk_scene_upload", ptr(tris), tris.shape[0], ptr(pos), ptr(attrs), pos.shape[0])
    ctx.call("pk_bvh_build", _lib.PK_BVH_SWEEP)
    nn, nt = C.c_uint32(), C.c_uint32()
    ctx.call("pk_bvh_info", C.byref(nn), C.byref(nt), None)
    assert (nn.value, nt.value) == (ref.nodes.shape[0], ref.tris.shape[0])
    nodes, leaf = np.zeros_like(ref.nodes), np.zeros_like(ref.tris)
    verts = np.zeros_like(ref.verts)
    ctx.call("pk_bvh_download", ptr(nodes), ptr(leaf), ptr(verts))
    assert np.array_equal(nodes, ref.nodes)
    assert np.array_equal(leaf, ref.tris)
    assert_bits_equal(verts, ref.verts, "vertices")


def test_sweep_build_refuses_a_point(ctx):
    """A node without surface area has no finite cost: refused, and the context builds again."""
    pos = np.zeros((3, 3))
    tris = np.array([[0, 1, 2, 0]], np.int32)
    attrs = np.zeros((3, 4), np.uint32)
    ctx.call("pk_scene_upload", ptr(tris), 1, ptr(pos), ptr(attrs), 3)
    with pytest.raises(_lib.PikeError):
        ctx.call("pk_bvh_build", _lib.PK_BVH_SWEEP)
    pos, tris = soup(40, 1)
    attrs = np.zeros((120, 4), np.uint32)
    ctx.call("pk_scene_upload", ptr(tris), 40, ptr(np.ascontiguousarray(pos)), ptr(attrs), 120)
    ctx.call("pk_bvh_build", _lib.PK_BVH_SWEEP)


@pytest.mark.parametrize("w,h,kind", [(2, 1, "log"), (2047, 1, "log"), (2048, 1, "log"), (1, 2049, "log"),
                                      (128, 96, "log"), (3071, 1, "log"), (3072, 1, "log"), (1, 3073, "log"),
                                      (97, 64, "log"), (64, 64, "two"), (128, 64, "steep"), (96, 64, "constant")])
def test_env_tables_at_sort_tiles_and_bin_edges(ctx, oracle, w, h, kind):
    """Tiles of 2048 keys, 1 to 6 of them (a look-back reads 4); maps whose bin edges fall on ties (decided by the sequential walk)."""
    rng = np.random.default_rng(w * h)
    lum = {"log": lambda: np.exp(1.5 * rng.standard_normal((h, w))), "two": lambda: rng.integers(1, 3, (h, w)) * 1.0,
           "steep": lambda: 2.0 ** -rng.uniform(0, 60, (h, w)), "constant": lambda: np.ones((h, w))}[kind]()
    rgbe = np.ascontiguousarray(synth.rgbe_encode(np.repeat(lum[..., None], 3, axis=2)))
    try:
        ref = oracle.Env(rgbe)
    except Exception:  # a map the reference cannot sample is refused here too
        with pytest.raises(_lib.PikeError):
            ctx.call("pk_env_build", ptr(rgbe), w, h)
        return
    ctx.call("pk_env_build", ptr(rgbe), w, h)
    nb = C.c_uint32()
    ctx.call("pk_env_info", None, None, C.byref(nb))
    assert nb.value == ref.bins.shape[0]
    bins, coords, pdf = np.zeros_like(ref.bins), np.zeros_like(ref.coords), np.zeros_like(ref.pdf)
    ctx.call("pk_env_download", ptr(bins), ptr(coords), ptr(pdf))
    assert np.array_equal(bins, ref.bins) and np.array_equal(coords, ref.coords)
    assert_bits_equal(pdf, ref.pdf, "pdf")


@pytest.mark.parametrize("n", [1, 32, 1023, 1024, 1025, 2048, 2049, 20_000])
@pytest.mark.parametrize("any_hit", [False, True])
def test_queries_at_block_and_tile_edges(oracle, pk_built, n, any_hit):
    torch = pytest.importorskip("torch")
    src = synth.displaced_sphere_scene(subdivisions=4, width=8, height=8, env_size=(64, 32))
    pair = Pair(src, oracle)
    rng = np.random.default_rng(n)
    o, d = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    o[:, :3] = rng.uniform(-0.9, 0.9, (n, 3))
    d[:, :3] = rng.normal(size=(n, 3))
    ref = pair.P.r.trace_rays(np.concatenate([o, d], axis=1), any_hit=any_hit)
    for call in ("pk_cast_rays", "pk_cast_rays_noalloc"):
        to, td = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
        hits = torch.full((n, 4), -7, dtype=torch.int32, device="cuda")
        idx = torch.full((n,), -7, dtype=torch.int32, device="cuda")
        cnt = torch.full((1,), -7, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        pair.ctx.call(call, to.data_ptr(), td.data_ptr(), n, int(any_hit), hits.data_ptr(), idx.data_ptr(),
                      cnt.data_ptr())
        got = hits.cpu().numpy().view(np.uint32)
        hit = ref[:, 1] != 0xFFFFFFFF
        assert np.array_equal(got[:, 1], ref[:, 1])
        assert np.array_equal(got[hit, 0], ref[hit, 0]) and np.array_equal(got[hit, 2], ref[hit, 2])
        k = int(cnt.item())
        assert np.array_equal(idx[:k].cpu().numpy(), np.flatnonzero(hit))


@pytest.mark.parametrize("w,h", [(33, 31), (32, 32), (41, 25), (67, 61), (1024, 1024)])
def test_frames_at_compaction_tiles(oracle, pk_built, w, h):
    """Tiles of 1024 rays, of 4096 from 2^20 rays on; fused frames and the pass path."""
    bounces = 2 if w * h > 100_000 else 4
    src = synth.small_scene(width=w, height=h, bounces=bounces)
    pair = Pair(src, oracle)
    pair.set_render_state(0)
    pair.P.r.tick(bounces)
    want = pair.P.r.accum()
    c = pair.ctx
    for in_flight in (1, 4):
        c.call("pk_set_frames_in_flight", in_flight)
        c.call("pk_set_render_state", 0, 0.0)
        c.call("pk_render_frame", bounces)
        c.call("pk_sync")
        assert_bits_equal(pair.image("accum"), want, f"{in_flight} in flight")
    c.call("pk_set_render_state", 0, 0.0)
    for name in ["clear_color", "clear_hits_misses", "clear_rays", "camera"] + ["trace", "shade_hit", "trace_shadow",
                                                                             "shade_miss"] * bounces + ["accumulate"]:
        c.call("pk_" + name)
    c.call("pk_sync")
    assert_bits_equal(pair.image("accum"), want, "pass by pass")


def test_paths_in_chunks(pk_built):
    """More paths than a chunk (2^22) holds: the image and the gradients are those of the samples cut in two."""
    torch = pytest.importorskip("torch")
    from pike_gb300.diff import DiffScene
    src = synth.displaced_sphere_scene(subdivisions=3, width=64, height=64, env_size=(64, 32))
    spp = 1100  # 64 * 64 * 1100 = 4.5M paths
    whole = DiffScene(src, 64, 64, spp=spp, depth=3)
    half = DiffScene(src, 64, 64, spp=spp // 2, depth=3)
    albedo, rough, env = whole.source_params(env_size=(64, 32))
    for s in (whole, half):
        s.set_env_sampling(env)
    image = whole.render(albedo, rough, env, seed=0)
    rays = whole.rays()
    parts, n = [], 0
    for k in (0, 1):
        parts.append(half.render(albedo, rough, env, seed=k))
        n += half.rays()
    assert rays == n
    # sums of 1100 binary32 values in another grouping: 1100 * 2^-24 relative
    mean = (parts[0].double() + parts[1].double()) / 2
    assert ((image.double() - mean).abs() <= 7e-5 * (mean.abs() + 1e-3)).all()
    d = torch.ones_like(image)
    g = whole.backward(albedo, rough, env, d, seed=0)
    h = [half.backward(albedo, rough, env, d / 2, seed=k) for k in (0, 1)]
    for name, a, b0, b1 in zip(("albedo", "rough", "env"), g, *h):
        b = b0 + b1
        assert (a - b).abs().max() <= 1e-4 * b.abs().max(), name


@pytest.mark.parametrize("change", [
    dict(), dict(apertureSize=0.05), dict(bokeh=-1.0), dict(bokeh=0.0), dict(focalDepth=float("inf")),
    dict(pos=[-0.0, 1.5, 4.0]), dict(pos=[0.0, -0.0, 4.0], apertureSize=0.0), dict(dir=[0.0, 1.0, 0.0]),
    dict(fov=3.0, distortion=0.4)], ids=str)
def test_camera_rays_with_and_without_a_lens(oracle, pk_built, change):
    """A zero aperture leaves the lens out where that changes no bit, and only there."""
    src = synth.small_scene(width=33, height=17)
    pair = Pair(src, oracle)
    pair.set_camera(dict(src.camera_state(), **change))
    pair.set_render_state(3)
    P = pair.P.r
    for name in ("clear_color", "clear_hits_misses", "clear_rays"):
        pair.ctx.call("pk_" + name)
    P.begin_frame()
    pair.ctx.call("pk_camera")
    P.camera()
    n = P.counters()["num_rays"]
    assert_bits_equal_nan(pair.rays(_lib.PK_QUEUE_RAYS, 0, n), P.rays(0, n), "camera rays")


@pytest.mark.parametrize("theta", [0.0, -0.5, -3.9, 2.7, 1.0e4, 3.0e6])
def test_environment_lookup_wraps(oracle, pk_built, theta):
    """Repeat addressing of the rotated map: inside it, some turns away on both
    sides, and beyond 2^20 texels, where the integer remainder takes over."""
    src = synth.displaced_sphere_scene(subdivisions=3, width=64, height=40, env_size=(67, 31))
    pair = Pair(src, oracle)
    pair.set_render_state(0, theta)
    P = pair.P.r
    for name in ("clear_color", "clear_hits_misses", "clear_rays"):
        pair.ctx.call("pk_" + name)
    P.begin_frame()
    for name in ("camera", "trace", "shade_hit", "trace_shadow", "shade_miss", "accumulate"):
        pair.ctx.call("pk_" + name)
        getattr(P, name)()
    want = P.accum()
    assert_bits_equal(pair.image("accum"), want, "pass by pass")
    pair.ctx.call("pk_set_render_state", 0, theta)
    pair.ctx.call("pk_render_frame", 1)
    pair.ctx.call("pk_sync")
    assert_bits_equal(pair.image("accum"), want, "fused")


@pytest.mark.parametrize("capacity", [(1 << 19) - 128, 1 << 19, 1 << 20])
def test_queue_capacity_changes_no_bit(oracle, pk_built, capacity):
    """The same 2046 rays in queues on both sides of the lines where shading and compaction change form."""
    src = synth.small_scene(width=66, height=31)
    pair = Pair(src, oracle)
    pair.set_render_state(0)
    pair.P.r.tick(4)
    want = pair.P.r.accum()
    pair.ctx.call("pk_configure", src.width, src.height, capacity)
    pair.ctx.call("pk_set_camera", C.byref(camera_struct(src.camera_state())))
    pair.ctx.call("pk_set_render_state", 0, 0.0)
    pair.ctx.call("pk_render_frame", 4)
    pair.ctx.call("pk_sync")
    assert_bits_equal(pair.image("accum"), want, "fused")


def test_batch_readback_in_parts(pk_built):
    """A request of more than the 2^20 pixels that are read back at a time: the
    pixels whose camera ray misses have the drop-in's bits (shading seeds differ)."""
    from pike_gb300.batch import Batch, Request, scene_context
    w, h = 1100, 1000
    src = synth.small_scene(width=w, height=h)
    ctx, cam = scene_context(src), dict(src.camera_state(), dir=[0.0, 0.4, 0.9165151])  # up: sky below as well
    batch = Batch([ctx])
    batch.set_requests([Request(scene=0, width=w, height=h, spp=1, depth=1, camera=cam)])
    batch.render(1)
    got = batch.image(0)
    ctx.call("pk_configure", w, h, w * h)
    ctx.call("pk_set_camera", C.byref(camera_struct(cam)))
    ctx.call("pk_set_render_state", 0, 0.0)
    want = np.zeros((h, w, 4), np.float32)
    for name in ("clear_color", "clear_hits_misses", "clear_rays", "camera", "trace"):
        ctx.call("pk_" + name)
    n = np.zeros(8, np.uint32)
    ctx.call("pk_read_counters", ptr(n))
    hits = np.zeros((int(n[1]), 16), np.uint32)
    ctx.call("pk_read_hits", 0, hits.shape[0], ptr(hits))
    ctx.call("pk_set_render_state", 0, 0.0)
    ctx.call("pk_render_frame", 1)
    ctx.call("pk_read_accum", ptr(want))
    miss = np.ones(w * h, bool)
    miss[hits[:, 15] & 0x0FFFFFFF] = False
    assert miss[: 1 << 20].any() and miss[1 << 20:].any()
    assert np.array_equal(got.reshape(-1, 4)[miss, :3].view(np.uint32), want.reshape(-1, 4)[miss, :3].view(np.uint32))
