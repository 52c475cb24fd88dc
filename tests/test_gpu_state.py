"""What one call leaves behind for the next on the same context."""
import pytest

from pike_gb300 import _lib, synth

from helpers import Pair, assert_bits_equal

pytestmark = pytest.mark.gpu


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
