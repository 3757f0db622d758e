"""Swish + FP4 output of a GEMM (the feed-forward up-projection) against the stand-alone quantizer on the same GEMM's fp32 output:
each warp takes 64 columns of one half of the wide tile, so the edges are row blocks and column counts that end in a first half."""

import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def _unsigned_zeros(codes):
    lo, hi = codes & 0x0F, codes & 0xF0
    return torch.where((lo & 7) == 0, 0, lo) | torch.where((hi & 0x70) == 0, 0, hi)


@pytest.mark.parametrize("fmt", ["mx32", "nv16"])
@pytest.mark.parametrize("M", [1, 127, 128, 129, 300, 148 * 128 + 1])
def test_swish_codes_are_the_quantized_fp32_output(fmt, M):
    from velox_voice_b200 import _lib, ops
    from velox_voice_b200.linear import PackedLinear

    g = torch.Generator(device="cuda").manual_seed(M)
    am = torch.tensor([4.0], device="cuda") if fmt == "nv16" else None
    for N, K, bias in ((2048, 512, True), (128, 256, True), (384, 512, False), (512, 1024, True), (640, 2048, True)):
        x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
        x[0, : K // 2] = 0
        b = 0.1 * torch.randn(N, generator=g, device="cuda") if bias else None
        lin = PackedLinear(0.05 * torch.randn(N, K, generator=g, device="cuda"), b, fmt)
        a = ops.quantize(x, fmt)
        want = ops.quantize(lin(a, act="swish", out_dtype=torch.float32), fmt, amax_t=am, natural=True)
        got = lin(a, act="swish", out_fmt=fmt, out_amax=am)
        assert torch.equal(_unsigned_zeros(got.codes), _unsigned_zeros(want.codes)), (N, K)
        assert torch.equal(got.sf, want.sf), (N, K)
        # the scales in the natural layout as well, through the C ABI
        d, keep = ops._gemm_desc(a, lin.q, lin.bias)
        codes, sf, scales = torch.empty_like(want.codes), torch.full_like(want.sf, 255), torch.full_like(want.scales, 255)
        d.epilogue, d.out_dtype, d.out, d.ldo = _lib.EPI_BIAS_SWISH, _lib.DT_FP4, codes.data_ptr(), N // 2
        d.out_fmt, d.out_scales, d.out_scales_sf = a.fmt, scales.data_ptr(), sf.data_ptr()
        if am is not None:
            d.out_amax = am.data_ptr()
        _lib.check(_lib.load().vx_bsgemm(C.byref(d), torch.cuda.current_stream().cuda_stream), "vx_bsgemm")
        assert torch.equal(codes, got.codes) and torch.equal(sf, got.sf) and torch.equal(scales, want.scales)
    assert _lib.device_status() == 0
