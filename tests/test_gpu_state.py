"""What one call leaves behind for the next on the same context, and builds at
scales where the reference's own arithmetic gives out."""
import ctypes as C

import numpy as np
import pytest

from pike_gb300 import _lib, synth
from pike_gb300._lib import Context, ptr

import test_gpu_edges
from helpers import Pair, assert_bits_equal, camera_struct

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(pk_built):
    return Context(0)


def pass_by_pass(pair, bounces):
    c = pair.ctx
    c.call("pk_set_render_state", 0, 0.0)
    for name in ["clear_color", "clear_hits_misses", "clear_rays", "camera"] + ["trace", "shade_hit", "trace_shadow",
                                                                             "shade_miss"] * bounces + ["accumulate"]:
        c.call("pk_" + name)
    c.call("pk_sync")
    return pair.image("accum")


@pytest.mark.parametrize("mode", [_lib.PK_TRACE_PERSISTENT, _lib.PK_TRACE_PERSISTENT | _lib.PK_TRACE_COMPACT_RECORDS,
                                  _lib.PK_TRACE_PERSISTENT | _lib.PK_TRACE_WIDE,
                                  _lib.PK_TRACE_PERSISTENT | _lib.PK_TRACE_EXACT])
def test_passes_after_a_frame_of_the_chunked_schedule(oracle, pk_built, mode):
    """The shadow outcome bits of a fused frame must not reach a later pass."""
    src = synth.small_scene(width=96, height=64)
    used, fresh = Pair(src, oracle), Pair(src, oracle)
    used.ctx.call("pk_set_trace_mode", _lib.PK_TRACE_CHUNKED)
    used.set_render_state(0)
    used.ctx.call("pk_render_frame", 4)
    used.ctx.call("pk_sync")
    for p in (used, fresh):
        p.ctx.call("pk_set_trace_mode", mode)
    assert_bits_equal(pass_by_pass(used, 4), pass_by_pass(fresh, 4), f"mode {mode}")


def cast(ctx, n=64):
    torch = pytest.importorskip("torch")
    o, d = torch.zeros((n, 4), device="cuda"), torch.ones((n, 4), device="cuda")
    hits = torch.zeros((n, 4), dtype=torch.int32, device="cuda")
    idx, cnt = torch.zeros(n, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    for call in ("pk_cast_rays", "pk_cast_rays_noalloc"):
        ctx.call(call, o.data_ptr(), d.data_ptr(), n, 0, hits.data_ptr(), idx.data_ptr(), cnt.data_ptr())


@pytest.mark.parametrize("n", [511, 512, 513])
@pytest.mark.parametrize("any_hit", [False, True])
def test_queries_around_one_block(oracle, pk_built, n, any_hit):
    test_gpu_edges.test_queries_at_block_and_tile_edges(oracle, pk_built, n, any_hit)


def test_queries_beyond_the_kept_scratch(oracle, pk_built):
    """2^20 rays use the context's scratch, more take theirs from the pool: one query
    of both kinds and the same rays in two of the first."""
    torch = pytest.importorskip("torch")
    ctx = Pair(synth.small_scene(width=8, height=8), oracle).ctx
    n, half = (1 << 20) + 5, 1 << 19
    g = torch.Generator().manual_seed(1)
    o = torch.nn.functional.pad(torch.rand((n, 3), generator=g) * 1.8 - 0.9, (0, 1)).cuda()
    d = torch.nn.functional.pad(torch.randn((n, 3), generator=g), (0, 1)).cuda()

    def query(o, d):
        hits = torch.zeros((o.shape[0], 4), dtype=torch.int32, device="cuda")
        idx, cnt = torch.zeros(o.shape[0], dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        ctx.call("pk_cast_rays", o.data_ptr(), d.data_ptr(), o.shape[0], 0, hits.data_ptr(), idx.data_ptr(), cnt.data_ptr())
        return hits, idx[:cnt.item()]
    whole, a, b = query(o, d), query(o[:half], d[:half]), query(o[half:], d[half:])
    assert torch.equal(whole[0], torch.cat([a[0], b[0]]))
    assert torch.equal(whole[1], torch.cat([a[1], b[1] + half]))


def upload_bvh(ctx, nodes, tris, verts):
    ctx.call("pk_bvh_upload", ptr(nodes), nodes.shape[0], ptr(tris), tris.shape[0], ptr(verts), verts.shape[0])


def frame(pair, bounces=4):
    pair.ctx.call("pk_set_render_state", 0, 0.0)
    pair.ctx.call("pk_render_frame", bounces)
    pair.ctx.call("pk_sync")
    return pair.image("accum")


@pytest.mark.parametrize("mode", [_lib.PK_TRACE_PERSISTENT, _lib.PK_TRACE_PERSISTENT | _lib.PK_TRACE_WIDE,
                                  _lib.PK_TRACE_PERSISTENT | _lib.PK_TRACE_EXACT])
def test_refused_bvh_leaves_nothing_to_traverse(oracle, pk_built, mode):
    """A malformed upload over a BVH in use, with a captured frame: every traversal
    is refused until a sound BVH is there, and then gives the first image again."""
    src = synth.small_scene(width=64, height=48)
    pair = Pair(src, oracle)
    c, b = pair.ctx, pair.P.bvh
    c.call("pk_set_trace_mode", mode)
    want = frame(pair)
    bad = np.ascontiguousarray(b.nodes[:5]).copy()
    bad[0, :2] = (7, -1)  # a child outside the tree
    with pytest.raises(_lib.PikeError):
        upload_bvh(c, bad, np.ascontiguousarray(b.tris[:3]), b.verts)
    for call in (lambda: frame(pair), lambda: cast(c), lambda: c.call("pk_trace")):
        with pytest.raises(_lib.PikeError):
            call()
    upload_bvh(c, b.nodes, b.tris, b.verts)
    cast(c)
    assert_bits_equal(frame(pair), want, "after a sound upload")
    c.call("pk_bvh_build", _lib.PK_BVH_SWEEP)
    assert_bits_equal(frame(pair), want, "after a build")


@pytest.mark.parametrize("mode", [_lib.PK_TRACE_WIDE, _lib.PK_TRACE_EXACT])
def test_bvh_that_only_the_drop_in_records_hold(oracle, pk_built, mode):
    """Two parents of one pair of leaves: the drop-in's records hold that, a tree
    with each node reached once is needed for the others.  Refused there, usable here."""
    src = synth.small_scene(width=64, height=48)
    pair = Pair(src, oracle)
    c, b = pair.ctx, pair.P.bvh
    box = b.nodes[0, 2:]
    nodes = np.array([[1, -1, *box], [3, -1, *box], [3, -1, *box], [-1, (2 << 24) | 0, *box], [-1, (1 << 24) | 2, *box]],
                     np.int32)
    tris = np.ascontiguousarray(b.tris[:3])
    c.call("pk_set_trace_mode", _lib.PK_TRACE_PERSISTENT | mode)
    frame(pair)
    with pytest.raises(_lib.PikeError):
        upload_bvh(c, nodes, tris, b.verts)
    with pytest.raises(_lib.PikeError):
        frame(pair)
    cast(c)
    c.call("pk_set_trace_mode", _lib.PK_TRACE_PERSISTENT)
    got = frame(pair)
    c.call("pk_set_trace_mode", _lib.PK_TRACE_CHUNKED)
    assert_bits_equal(frame(pair), got, "the drop-in's records")


@pytest.mark.parametrize("lacks", ["materials", "attributes", "vertices"])
def test_paths_need_the_whole_scene(pk_built, lacks):
    """Differentiable and batched rendering refuse a BVH without materials or vertex
    attributes, as frames do.  Vertices beyond the attributes take the first one's there."""
    torch = pytest.importorskip("torch")
    from pike_gb300.batch import Batch, scene_context
    from pike_gb300.diff import DiffScene
    src = synth.small_scene(width=32, height=24)
    whole = DiffScene(src, 32, 24, spp=1, depth=2)
    params = whole.source_params(env_size=(32, 16))
    whole.render(*params)
    donor = scene_context(src)
    n, k = C.c_uint32(), C.c_uint32()
    donor.call("pk_bvh_info", C.byref(n), C.byref(k), None)
    nodes, tris = np.zeros((n.value, 5), np.int32), np.zeros((k.value, 4), np.int32)
    verts = np.zeros((src.pos.shape[0], 4), np.float32)
    donor.call("pk_bvh_download", ptr(nodes), ptr(tris), ptr(verts))
    ctx = Context(0)
    ctx.call("pk_configure", 32, 24, 32 * 24)
    if lacks != "materials":
        ctx.call("pk_materials_set", ptr(np.ascontiguousarray(src.materials, np.float64)), src.materials.shape[0])
    if lacks != "attributes":
        m = 3 if lacks == "vertices" else src.pos.shape[0]
        ctx.call("pk_scene_upload", ptr(np.array([[0, 1, 2, 0]], np.int32)), 1,
                 ptr(np.ascontiguousarray(src.pos[:m], np.float64)), ptr(np.zeros((m, 4), np.uint32)), m)
    upload_bvh(ctx, nodes, tris, verts)
    ctx.call("pk_env_build", ptr(src.env_rgbe), src.env_rgbe.shape[1], src.env_rgbe.shape[0])
    part = DiffScene.__new__(DiffScene)
    part.__dict__.update(whole.__dict__, ctx=ctx, env_shape=None)
    ctx.call("pk_set_camera", C.byref(camera_struct(whole.camera_state)))
    if lacks == "vertices":
        Batch([ctx])
        part.render(*params)
        part.backward(*params, torch.ones((24, 32, 4), device="cuda"))
        return
    with pytest.raises(_lib.PikeError):
        Batch([ctx])
    with pytest.raises(_lib.PikeError):
        part.render(*params)
    with pytest.raises(_lib.PikeError):
        part.backward(*params, torch.ones((24, 32, 4), device="cuda"))


@pytest.mark.parametrize("fn,div,signed", [(9, 127.0, True), (10, 255.0, False)])
def test_byte_decodes_of_every_position_and_pair(ctx, fn, div, signed):
    """Each byte position and each half of a packed decode, every value beside every
    other: the IEEE quotient (max(v / d, -1) when signed)."""
    v, u = (a.reshape(-1).astype(np.int32) for a in np.meshgrid(np.arange(256), np.arange(256)))
    got = np.zeros(v.size, np.float32)
    ctx.call("pk_math_eval", fn, ptr(v.view(np.float32)), ptr(u.view(np.float32)), ptr(got), v.size)
    want = (v.astype(np.int8) if signed else v).astype(np.float32) / np.float32(div)
    assert_bits_equal(got, np.maximum(want, np.float32(-1.0)), f"decode fn {fn}")


def test_env_tables_of_three_scan_levels(ctx, oracle):
    """More than 2^22 texels: the prefix sums behind the bins take a third level."""
    test_gpu_edges.test_env_tables_at_sort_tiles_and_bin_edges(ctx, oracle, 4099, 1025, "log")


def build_sweep(ctx, pos, tris):
    pos = np.ascontiguousarray(pos)
    attrs = np.zeros((pos.shape[0], 4), np.uint32)
    ctx.call("pk_scene_upload", ptr(tris), tris.shape[0], ptr(pos), ptr(attrs), pos.shape[0])
    ctx.call("pk_bvh_build", _lib.PK_BVH_SWEEP)


@pytest.mark.parametrize("n", [40, 700, 1500])
@pytest.mark.parametrize("exponent", [-175, -165, -160, -158, -150, -141, -139, 149, 151, 153, 154, 160, 170])
def test_sweep_build_where_areas_underflow_or_overflow(ctx, oracle, n, exponent):
    """Extents whose products leave the normal doubles: the reference's costs are
    then inexact or not finite, and the same trees have to come out, or the same refusals."""
    pos, tris = test_gpu_edges.soup(n, n, spread=10.0 ** exponent)
    try:
        ref = oracle.BVH(np.ascontiguousarray(pos), tris)
    except Exception:  # no finite split cost
        with pytest.raises(_lib.PikeError):
            build_sweep(ctx, pos, tris)
        return
    build_sweep(ctx, pos, tris)
    nn, nt = C.c_uint32(), C.c_uint32()
    ctx.call("pk_bvh_info", C.byref(nn), C.byref(nt), None)
    assert (nn.value, nt.value) == (ref.nodes.shape[0], ref.tris.shape[0])
    nodes, leaf = np.zeros_like(ref.nodes), np.zeros_like(ref.tris)
    ctx.call("pk_bvh_download", ptr(nodes), ptr(leaf), None)
    assert np.array_equal(nodes, ref.nodes) and np.array_equal(leaf, ref.tris)
