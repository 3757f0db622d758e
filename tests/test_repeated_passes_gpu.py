"""The same work repeated gives the same bytes, whatever overlaps what."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", ["mx32", "nv16", "fp8_1x128"])
@pytest.mark.parametrize("M,N", [(24000, 5538), (24000, 162), (24000, 290), (40000, 32), (30000, 416)])
def test_staged_stores_of_ragged_widths(fmt, M, N):
    """bf16 output through the staging buffers and TMA, with last column blocks that leave a warp one of its two chunks or
    none, against per-thread stores.  N = 5,538 (the CTC head): about one launch in twenty had rows of a 32-row block that
    held the values of a later tile."""
    from velox_voice_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(N)
    a = ops.quantize(torch.randn(M, 512, generator=g, device="cuda").bfloat16(), fmt)
    b = ops.quantize(0.05 * torch.randn(N, 512, generator=g, device="cuda"), fmt)
    bias = torch.randn(N, generator=g, device="cuda")
    want = ops.bsgemm(a, b, epilogue=ops.EPI_BIAS, bias=bias, direct_store=True)
    bad = 0
    for _ in range(20):
        outs = [ops.bsgemm(a, b, epilogue=ops.EPI_BIAS, bias=bias) for _ in range(8)]
        bad += sum(not torch.equal(o, want) for o in outs)
        del outs
    assert bad == 0, f"{bad} of 160 launches differ"


def expected(frames):
    """A stack, features, positions, and hidden states and logits of a pass in which the residual GEMMs, LayerNorms and quantizers run
    as separate kernels and the logits leave by per-thread stores."""
    from velox_voice_b200 import ops
    from velox_voice_b200.stack import ConformerLinearStack, StackConfig, make_weights

    cfg = StackConfig()
    stack = ConformerLinearStack(cfg, make_weights(cfg, seed=3))
    g = torch.Generator(device="cuda").manual_seed(frames)
    x = torch.randn(frames, cfg.d_model, generator=g, device="cuda").bfloat16()
    pos = torch.randn(frames, cfg.d_model, generator=g, device="cuda").bfloat16()
    stack.fuse_ln = False
    _, hidden = stack.forward(x.clone(), pos, return_hidden=True)
    torch.cuda.synchronize()
    q = ops.ln_quantize(hidden, *stack.ln["after"], cfg.eps, "mx32")
    want = ops.bsgemm(q, stack.p["ctc"].q, epilogue=ops.EPI_BIAS, bias=stack.p["ctc"].bias, direct_store=True)
    return stack, x, pos, hidden, want


@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("frames,passes", [(375, 400), (4800, 200), (21090, 200), (24000, 200)])
def test_passes_of_the_stack(frames, passes, fused):
    """Passes issued eight at a time without a pause between them, against a pass in which the residual GEMMs, LayerNorms and
    quantizers run as separate kernels and the logits leave by per-thread stores."""
    from velox_voice_b200 import _lib, ops

    stack, x, pos, hidden, want = expected(frames)
    stack.fuse_ln, stack.fuse_ln_min_frames = fused, 0
    bad = 0
    ops.reset_launch_count()
    for _ in range(passes // 8):
        outs = [stack.forward(x.clone(), pos, return_hidden=True) for _ in range(8)]
        bad += sum(not (torch.equal(o, want) and torch.equal(h, hidden)) for o, h in outs)
        del outs
    assert bad == 0, f"{bad} of {passes} passes differ"
    assert _lib.device_status() == 0
    lp = 1 if frames <= 4096 else 12
    assert ops.launch_count() == passes // 8 * 8 * (2 + lp + (12 * 8 if fused else 12 * 12) + 1)


@pytest.mark.parametrize("frames,passes", [(375, 400), (1920, 400), (4096, 200)])
def test_passes_in_one_launch(frames, passes):
    """The same where all blocks run in one launch (clusters of eight CTAs, all of them, and of four)."""
    from velox_voice_b200 import _lib, ops

    stack, x, pos, hidden, want = expected(frames)
    stack.fuse_ln = True
    bad = 0
    ops.reset_launch_count()
    for _ in range(passes // 8):
        outs = [stack.forward(x.clone(), pos, return_hidden=True) for _ in range(8)]
        bad += sum(not (torch.equal(o, want) and torch.equal(h, hidden)) for o, h in outs)
        del outs
    assert bad == 0, f"{bad} of {passes} passes differ"
    assert _lib.device_status() == 0
    assert ops.launch_count() == passes // 8 * 8 * 4  # positions (quantizer, projections), blocks, head
