"""The one-launch pass: argument checks without a device, and the rule for waits in front of warp-wide tensor-memory accesses."""

import ctypes as C
import re

from test_device_sources_cpu import source
from test_device_sources_cpu import test_waits_before_warp_wide_tensor_memory_accesses_end_in_a_vote as vote_rule
from velox_voice_b200 import _lib


def test_arguments_are_checked_before_any_launch():
    lib = _lib.load()
    assert lib.vx_conformer_pass(None, None) == -1
    desc = (C.c_int32 * 64)()
    desc[0] = 8  # struct_size
    assert lib.vx_conformer_pass(C.cast(desc, C.c_void_p), None) == -1 and b"struct_size" in lib.vx_last_error()


def test_shapes_it_covers():
    ok = _lib.load().vx_conformer_pass_supported
    assert ok(_lib.FMT_MX32, 512, 2048, 1024, 12) == 1 and ok(_lib.FMT_MX32, 512, 1024, 1024, 16) == 1
    for args in ((_lib.FMT_NV16, 512, 2048, 1024, 12), (_lib.FMT_MX32, 256, 2048, 1024, 12), (_lib.FMT_MX32, 512, 1536, 1024, 12),
                 (_lib.FMT_MX32, 512, 4096, 1024, 12), (_lib.FMT_MX32, 512, 2048, 512, 12), (_lib.FMT_MX32, 512, 2048, 1024, 17),
                 (_lib.FMT_MX32, 512, 2048, 1024, 0)):
        assert ok(*args) == 0


def test_waits_end_in_a_vote():
    vote_rule("vx_pass.cu", "conformer_pass_kernel(")


def test_a_line_for_the_fused_launches_takes_passes_off_the_one_launch():
    """``fuse_ln_min_frames`` chooses between separate and fused launches for passes of every length, whenever it is assigned."""
    from velox_voice_b200.stack import ConformerLinearStack

    stack = object.__new__(ConformerLinearStack)  # (the route only: a stack's weights need a GPU)
    stack.fuse_ln, stack.fuse_ln_min_frames = True, 4737
    stack.one_launch_frames = 4224
    assert [stack._route(t) for t in (1, 4224, 4225, 4736, 4737)] == [2, 2, 0, 0, 1]
    stack.fuse_ln_min_frames = 375
    assert [stack._route(t) for t in (1, 374, 375, 4224)] == [0, 0, 1, 1]
    stack.fuse_ln = False
    assert stack._route(375) == 0


def test_only_constant_weights_are_read_ahead_of_the_previous_launch():
    """The launch before may have written a bias or a LayerNorm parameter; the flag speaks of weights.  Whoever triggers the next
    launch has waited."""
    text = source("vx_pass.cu")
    assert re.search(r"if \(warp != PS_WARP_B\) {\s*pdl_wait\(\);\s*pdl_launch_dependents\(\);\s*} else if \(!p.b_const\) {\s*pdl_wait\(\);\s*}", text)
    assert text.count("pdl_launch_dependents()") == 1
