"""Quantizers that run in a GEMM's epilogue: the GLU output and the tail columns of a bf16 output, against the
stand-alone quantizer on the GEMM's own bf16 result (byte for byte), and the stack passes built on them."""

import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu

ROWS = (1, 127, 128, 129, 300, 148 * 128 + 1)  # edges of the 128-row tile, one row more than a round over the SMs


def _operands(M, N, K, fmt, seed, glu=False):
    from velox_voice_b200 import ops
    from velox_voice_b200.linear import PackedLinear

    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    x[0, : K // 2] = 0
    lin = PackedLinear(0.05 * torch.randn(N, K, generator=g, device="cuda"), 0.1 * torch.randn(N, generator=g, device="cuda"), fmt, glu=glu)
    return ops.quantize(x, fmt), lin


@pytest.mark.parametrize("fmt", ["mx32", "nv16"])
@pytest.mark.parametrize("M", ROWS)
def test_glu_output_quantized_in_the_epilogue(fmt, M):
    from velox_voice_b200 import ops

    am = torch.tensor([2.5], device="cuda") if fmt == "nv16" else None
    for N, K in ((1024, 512), (256, 256), (512, 1024)):
        a, lin = _operands(M, N, K, fmt, M + N, glu=True)
        want = ops.quantize(lin(a), fmt, amax_t=am)
        got = lin(a, out_fmt=fmt, out_amax=am)
        assert got.k == N // 2 and torch.equal(got.codes, want.codes)
        assert torch.equal(got.sf, want.sf)


@pytest.mark.parametrize("fmt", ["mx32", "nv16"])
@pytest.mark.parametrize("M", ROWS)
def test_tail_columns_quantized_in_the_epilogue(fmt, M):
    from velox_voice_b200 import _lib, ops

    am = torch.tensor([2.5], device="cuda") if fmt == "nv16" else None
    for N, K, c0 in ((1536, 512, 1024), (512, 512, 0), (768, 2048, 512)):
        a, lin = _operands(M, N, K, fmt, M + N + c0)
        want_out = lin(a)
        want = ops.quantize(want_out[:, c0:], fmt, amax_t=am)
        d, keep = ops._gemm_desc(a, lin.q, lin.bias)
        out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
        codes = torch.empty(M, (N - c0) // 2, dtype=torch.uint8, device="cuda")
        sf = torch.full_like(want.sf, 255)
        d.epilogue, d.out_dtype, d.out, d.ldo = _lib.EPI_BIAS, _lib.DT_BF16, out.data_ptr(), N
        d.flags, d.out_fmt, d.quant_col0 = _lib.GEMM_QUANT_TAIL, a.fmt, c0
        d.out_scales, d.out_scales_sf = codes.data_ptr(), sf.data_ptr()
        if am is not None:
            d.out_amax = am.data_ptr()
        _lib.check(_lib.load().vx_bsgemm(C.byref(d), torch.cuda.current_stream().cuda_stream), "vx_bsgemm")
        assert torch.equal(out, want_out) and torch.equal(codes, want.codes)
        assert torch.equal(sf, want.sf)


@pytest.mark.parametrize("T", [1, 300, 4096, 4097])
def test_stack_source_and_batched_positions(T):
    """`source` leaves the features alone and gives the same logits; 4,096 positions run all blocks' projections in
    one launch, 4,097 one by one."""
    from velox_voice_b200 import ops
    from velox_voice_b200.stack import ConformerLinearStack, StackConfig, make_weights

    stack = ConformerLinearStack(StackConfig(blocks=2), make_weights(StackConfig(blocks=2), seed=3))
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, 512, generator=g, device="cuda").bfloat16()
    pos = torch.randn(T, 512, generator=g, device="cuda").bfloat16()
    work, kept = torch.empty_like(x), x.clone()
    got = stack.forward(work, pos, source=x)
    assert torch.equal(x, kept)
    ops.reset_launch_count()
    want = stack.forward(x, pos)
    n_pos = ops.launch_count()
    assert torch.equal(got, want) and torch.equal(work, x)
    ops.reset_launch_count()
    stack.forward(kept, None)
    assert n_pos - ops.launch_count() == (2 if T <= 4096 else 3)  # quantizer + one or two projections
