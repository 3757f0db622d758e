"""FP8 GLU GEMM: the warps of the gate columns pass sigmoid(gate) to those of the value columns; row scales are fetched a
round (four 128-wide K blocks) ahead.  Sizes at the edges of both: one row, a ragged last tile, several tiles per CTA
(the hand-over is reused), rounds of one, three, four and four + one K blocks, with and without bias."""

import pytest
import torch

from oracle import formats as F
from oracle import gemm as G

pytestmark = pytest.mark.gpu

# bf16 rounding of the result (2^-9) and as much again for the accumulation on the tensor core and the sigmoid, of the maximum
TOL = 2.0**-8


@pytest.mark.parametrize("M,N,K,with_bias", [(1, 128, 128, True), (129, 256, 384, True), (384, 512, 512, False),
                                             (5000, 1024, 512, True), (2500, 1024, 640, True), (300, 128, 1024, False)])
def test_fp8_glu(M, N, K, with_bias):
    from velox_voice_b200 import _lib, ops
    from velox_voice_b200.linear import glu_interleave_index, glu_tile

    torch.manual_seed(M + K)
    fmt = F.FMT_FP8_1X128
    x = torch.randn(M, K, device="cuda").bfloat16()
    w = (0.1 * torch.randn(N, K, device="cuda")).bfloat16()
    bias = torch.randn(N, device="cuda") if with_bias else torch.zeros(N, device="cuda")
    idx = glu_interleave_index(N, "cuda", glu_tile(fmt))
    a, b, b_plain = ops.quantize(x, fmt), ops.quantize(w[idx].contiguous(), fmt), ops.quantize(w, fmt)
    out = ops.bsgemm(a, b, epilogue=G.EPI_BIAS_GLU, bias=bias[idx].contiguous() if with_bias else None, out_dtype=torch.bfloat16)
    y = G.gemm_ref(fmt, a.codes.cpu().numpy(), a.scales.cpu().numpy(), b_plain.codes.cpu().numpy(), b_plain.scales.cpu().numpy())
    ref = torch.from_numpy(G.epilogue_ref(y, G.EPI_BIAS_GLU, bias.cpu().numpy())).float()
    got = out.float().cpu()
    assert got.shape == (M, N // 2)
    assert ((got - ref).abs().max() / ref.abs().max()).item() < TOL
    assert _lib.device_status() == 0
