"""Run by test_gpu_lookback.py with the path of a library whose look-backs can be
made to give up: every builder has to answer with the timeout and leave the
context fit for the next call."""
import ctypes as C
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))

import numpy as np  # noqa: E402

from pike_gb300 import _lib, synth  # noqa: E402
from pike_gb300._lib import Context, PikeError, ptr  # noqa: E402

from test_gpu_edges import soup  # noqa: E402

L = _lib.load(sys.argv[1])
SCAN, SORT, ALL = 0, 1, 0xFFFFFFFF


def gives_up(kind, lo, hi):
    assert L.pk_test_gives_up(kind, C.c_uint32(lo), C.c_uint32(hi)) == 0


def expect_timeout(call, what):
    try:
        call()
    except PikeError as e:
        assert e.code == _lib.PK_ERR_CUDA and "look-back" in str(e), f"{what}: {e}"
        return
    raise AssertionError(f"{what}: no error")


def bvh(ctx):
    n, k = C.c_uint32(), C.c_uint32()
    ctx.call("pk_bvh_info", C.byref(n), C.byref(k), None)
    nodes, tris = np.zeros((n.value, 5), np.int32), np.zeros((k.value, 4), np.int32)
    verts = np.zeros((3 * k.value, 4), np.float32)
    ctx.call("pk_bvh_download", ptr(nodes), ptr(tris), ptr(verts))
    return nodes, tris, verts


def tree_level_sizes(nodes):
    level, out = np.array([0]), []
    while level.size:
        out.append(level.size)
        inner = level[nodes[level, 1] <= -1]
        level = (nodes[inner, 0][:, None] + np.arange(2)).reshape(-1)
    return out


def wide_level_sizes(rec):
    level, out = np.array([0]), []
    while level.size:
        out.append(level.size)
        r = rec[level]
        count = np.array([bin(m).count("1") for m in r[:, 3] >> 24])
        level = np.concatenate([np.arange(b, b + k) for b, k in zip(r[:, 4], count)] or [np.zeros(0, np.int64)]).astype(np.int64)
    return out


def main():
    ctx = Context(0)
    ctx.call("pk_configure", 16, 16, 256)
    pos, tris = soup(60_000, 7)
    pos = np.ascontiguousarray(pos)
    ctx.call("pk_scene_upload", ptr(tris), tris.shape[0], ptr(pos), ptr(np.zeros((pos.shape[0], 4), np.uint32)), pos.shape[0])
    sweep = lambda: ctx.call("pk_bvh_build", _lib.PK_BVH_SWEEP)
    sweep()
    first = bvh(ctx)
    n = first[0].shape[0]

    for kind in (SORT, SCAN):  # the triangle sort; the ranks of the subtrees
        gives_up(kind, 0, 100_000)
        expect_timeout(sweep, f"sweep build {kind}")
        assert all(np.array_equal(a, b) for a, b in zip(bvh(ctx), first))  # the BVH before stays
        gives_up(kind, 0, 0)
        sweep()
        assert all(np.array_equal(a, b) for a, b in zip(bvh(ctx), first))
    gives_up(SCAN, 0, 100_000)
    expect_timeout(lambda: ctx.call("pk_bvh_build", _lib.PK_BVH_BINNED), "binned build")
    gives_up(SCAN, 0, 0)

    upload = lambda: ctx.call("pk_bvh_upload", ptr(first[0]), n, ptr(first[1]), first[1].shape[0], ptr(first[2]),
                              first[2].shape[0])
    gives_up(SCAN, n, n + 1)
    expect_timeout(upload, "upload")
    try:
        bvh(ctx)
        raise AssertionError("a BVH without records counts as there")
    except PikeError:
        pass
    gives_up(SCAN, 0, 0)
    upload()

    wide = _lib.PK_TRACE_PERSISTENT | _lib.PK_TRACE_WIDE
    exact = _lib.PK_TRACE_PERSISTENT | _lib.PK_TRACE_EXACT
    levels = tree_level_sizes(first[0])
    gives_up(SCAN, 2049, n)  # the levels of the tree
    assert max(levels) > 2048
    for mode in (wide, exact):
        expect_timeout(lambda: ctx.call("pk_set_trace_mode", mode), f"tree levels {mode}")
    gives_up(SCAN, n, n + 1)  # the ranks of the inner nodes
    expect_timeout(lambda: ctx.call("pk_set_trace_mode", exact), "exact records")
    gives_up(SCAN, 0, 0)
    ctx.call("pk_set_trace_mode", exact)
    ctx.call("pk_set_trace_mode", wide)
    nw, depth = C.c_uint32(), C.c_uint32()
    ctx.call("pk_wide_info", C.byref(nw), C.byref(depth))
    rec = np.zeros((nw.value, 20), np.uint32)
    ctx.call("pk_wide_download", ptr(rec), None)
    sizes = [s for s in wide_level_sizes(rec) if s > 2048 and s not in levels]
    assert sizes and sum(wide_level_sizes(rec)) == nw.value
    gives_up(SCAN, sizes[0], sizes[0] + 1)
    expect_timeout(upload, "wide BVH")  # builds the wide tree of the set mode
    gives_up(SCAN, 0, 0)
    upload()
    again = np.zeros_like(rec)
    ctx.call("pk_wide_download", ptr(again), None)
    assert np.array_equal(again, rec)

    rgb = np.exp(np.random.default_rng(1).standard_normal((96, 128, 1))) * np.ones(3)
    rgbe = np.ascontiguousarray(synth.rgbe_encode(rgb))
    env = lambda: ctx.call("pk_env_build", ptr(rgbe), 128, 96)
    alias = lambda: ctx.call("pk_set_env_sampling", _lib.PK_ENV_ALIAS)
    env()
    gives_up(SCAN, 0, ALL)
    expect_timeout(alias, "alias table")
    gives_up(SCAN, 0, 0)
    alias()
    gives_up(SORT, 0, ALL)
    expect_timeout(env, "environment tables")
    import torch
    t = torch.tensor(rgb, dtype=torch.float32, device="cuda").contiguous()
    torch.cuda.synchronize()
    sampling = lambda: ctx.call("pk_diff_set_env_sampling", C.c_void_p(t.data_ptr()), 128, 96)
    expect_timeout(sampling, "sampling tables")
    gives_up(SORT, 0, 0)
    env()
    sampling()
    print("ok")


main()
