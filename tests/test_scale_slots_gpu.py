"""NVFP4 residual GEMM whose scale factors go through two slots of their own (wide tile, long K) against the narrow tile, which
has them in its ring: the same products in the same order, so equal bytes.  Edges: a part stage of K, a last column block with one
scale-factor tile, several tiles per CTA, and, where a short K is streamed on request, one to four stages a tile for three slots of tiles and two
of scale factors, whose turns then run across the tiles."""

import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [1280, 1312, 1536, 2048, 4096])
@pytest.mark.parametrize("M,N", [(1, 512), (129, 384), (300, 512), (74 * 128 * 2 + 1, 512), (40 * 128, 1152)])
def test_wide_tile_equals_the_narrow_one(M, N, K):
    _compare(M, N, K, 4)


@pytest.mark.parametrize("K", [256, 288, 512, 768, 1024])
@pytest.mark.parametrize("M,N", [(1, 512), (129, 384), (300, 512), (74 * 128 * 2 + 1, 512), (40 * 128, 1152), (24000, 512)])
def test_streamed_short_k(M, N, K):
    _compare(M, N, K, 4 | 2)


def _compare(M, N, K, wide_flags):
    from velox_voice_b200 import _lib, ops
    from velox_voice_b200.linear import PackedLinear

    g = torch.Generator(device="cuda").manual_seed(M + K)
    lin = PackedLinear(0.05 * torch.randn(N, K, generator=g, device="cuda"), 0.1 * torch.randn(N, generator=g, device="cuda"), "nv16")
    a = ops.quantize(torch.randn(M, K, generator=g, device="cuda").bfloat16(), "nv16")
    res = torch.randn(M, N, generator=g, device="cuda").bfloat16()
    outs = []
    for flags in (wide_flags, 8):  # wide, narrow
        d, keep = ops._gemm_desc(a, lin.q, lin.bias)
        out = torch.full_like(res, float("nan"))
        d.epilogue, d.out_dtype, d.out, d.ldo, d.flags = _lib.EPI_BIAS_RESIDUAL, _lib.DT_BF16, out.data_ptr(), N, flags
        d.residual, d.residual_dtype, d.ldr, d.alpha = res.data_ptr(), _lib.DT_BF16, N, 0.5
        _lib.check(_lib.load().vx_bsgemm(C.byref(d), torch.cuda.current_stream().cuda_stream), "vx_bsgemm")
        outs.append(out)
    assert torch.equal(outs[0].view(torch.int16), outs[1].view(torch.int16))
    assert _lib.device_status() == 0
