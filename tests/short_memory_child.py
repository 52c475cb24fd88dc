"""Run by test_gpu_short_memory.py with the path of a library whose device
allocations fail on demand."""
import ctypes as C
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))

import numpy as np  # noqa: E402

from pike_gb300 import _lib, synth  # noqa: E402
from pike_gb300._lib import PikeError, ptr  # noqa: E402
from pike_gb300.batch import scene_context  # noqa: E402
from helpers import camera_struct  # noqa: E402

L = _lib.load(sys.argv[1])
L.pk_test_memory.argtypes = [C.c_size_t, C.c_int]
L.pk_test_memory.restype = None
NONE = C.c_size_t(-1).value


def memory(limit=NONE, fail_next=0):
    L.pk_test_memory(limit, fail_next)


def refused(call, code=None):
    try:
        call()
    except PikeError as e:
        assert code is None or e.code == code, str(e)
        return
    raise AssertionError("no error")


def pools(src):
    """One failure: what the pools hold is given back and the call goes on."""
    ctx = scene_context(src)
    n = C.c_uint32()
    ctx.call("pk_bvh_info", C.byref(n), None, None)
    for call in (lambda: ctx.call("pk_bvh_build", _lib.PK_BVH_SWEEP),  # from the pool first
                 lambda: ctx.call("pk_configure", 512, 512, 1 << 18)):  # from the device
        memory(fail_next=1)
        call()
        assert L.pk_test_memory_failed() == 1 and L.pk_test_memory_trims() >= 1
    memory()
    m = C.c_uint32()
    ctx.call("pk_bvh_info", C.byref(m), None, None)
    assert m.value == n.value


def frame(ctx, src, w, h):
    ctx.call("pk_configure", w, h, w * h)
    ctx.call("pk_set_camera", C.byref(camera_struct(src.camera_state())))
    ctx.call("pk_set_render_state", 0, 0.0)
    ctx.call("pk_render_frame", 3)
    out = np.zeros((h, w, 4), np.float32)
    ctx.call("pk_read_accum", ptr(out))
    ctx.call("pk_sync")
    return out


def replaced(src):
    """An allocation that fails for good: an error, nothing half-replaced in use, and the same results afterwards."""
    ctx = scene_context(src)
    want = frame(ctx, src, 64, 48)
    render = lambda: ctx.call("pk_render_frame", 3)
    tris = np.ascontiguousarray(src.tris, np.int32)
    pos = np.ascontiguousarray(src.pos, np.float64)
    mats = np.ascontiguousarray(src.materials, np.float64)
    more = np.zeros((pos.shape[0] * 40, 3))
    attrs = np.zeros((more.shape[0], 4), np.uint32)
    env, big = np.ascontiguousarray(src.env_rgbe), np.full((1024, 512, 4), 128, np.uint8)
    tr = np.zeros(3)

    def scene():
        ctx.call("pk_scene_flatten", ptr(pos), ptr(np.ascontiguousarray(src.normal)), ptr(np.ascontiguousarray(src.tangent)),
                 ptr(np.ascontiguousarray(src.uv)), pos.shape[0], ptr(tris), tris.shape[0], 1.0, ptr(tr))
        ctx.call("pk_bvh_build", _lib.PK_BVH_SWEEP)

    for fails, mend in (
            (lambda: ctx.call("pk_configure", 1024, 1024, 1 << 20), lambda: None),
            (lambda: ctx.call("pk_scene_upload", ptr(tris), tris.shape[0], ptr(more), ptr(attrs), more.shape[0]), scene),
            (lambda: ctx.call("pk_env_build", ptr(big), 512, 1024),
             lambda: ctx.call("pk_env_build", ptr(env), env.shape[1], env.shape[0])),
            (lambda: ctx.call("pk_atlas_upload", ptr(big), 512, 2), lambda: ctx.call("pk_materials_set", ptr(mats), mats.shape[0]))):
        memory(limit=200_000)
        refused(fails, _lib.PK_ERR_CUDA)
        memory()
        refused(render)
        mend()
        got = frame(ctx, src, 64, 48)
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


def paths(src):
    """Differentiable rendering with less workspace than it would take: smaller chunks,
    the same image and the same gradients (sums in another grouping)."""
    import torch
    from pike_gb300.diff import DiffScene
    w, h, spp = 96, 64, 24
    s = DiffScene(src, w, h, spp=spp, depth=3)
    params = s.source_params(env_size=(64, 32))
    s.set_env_sampling(params[2])
    d = torch.rand((h, w, 4), device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    image, rays = s.render(*params), s.rays()
    grads = s.backward(*params, d)
    for limit in (20_000_000, 8_000_000):  # 147,456 paths take 31 MB forward, 67 MB backward
        t = DiffScene(src, w, h, spp=spp, depth=3)
        t.set_env_sampling(params[2])
        memory(limit=limit)
        got = t.render(*params)
        assert L.pk_test_memory_failed() >= 2  # once more after the pools were given back, then halved
        assert torch.equal(got.view(torch.int32), image.view(torch.int32)) and t.rays() == rays
        assert torch.equal(t.render(*params).view(torch.int32), image.view(torch.int32))  # the space is kept
        for name, a, b in zip(("albedo", "rough", "env"), t.backward(*params, d), grads):
            assert (a - b).abs().max() <= 1e-4 * b.abs().max(), name
        assert t.rays() == rays
        memory()
        del t
    t = DiffScene(src, w, h, spp=spp, depth=3)
    t.set_env_sampling(params[2])
    memory(limit=1000)
    refused(lambda: t.render(*params), _lib.PK_ERR_CUDA)
    memory()
    assert torch.equal(t.render(*params).view(torch.int32), image.view(torch.int32))


if __name__ == "__main__":
    source = synth.small_scene(width=64, height=48)
    pools(source)
    replaced(source)
    paths(source)
    print("ok")
