"""Residual epilogue: the fp32 result (bias added one value at a time) rounds to the bf16 result (pairs of values), whose residual comes by TMA."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", ["mx32", "nv16", "fp8_1x128"])
@pytest.mark.parametrize("M", [1, 129, 300, 24001])
@pytest.mark.parametrize("N,K", [(512, 512), (200, 512), (512, 2048)])
def test_fp32_and_bf16_results_agree(fmt, M, N, K):
    from velox_voice_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = ops.quantize(torch.randn(M, K, generator=g, device="cuda").bfloat16(), fmt)
    b = ops.quantize(0.05 * torch.randn(N, K, generator=g, device="cuda"), fmt)
    bias, res = torch.randn(N, generator=g, device="cuda"), torch.randn(M, N, generator=g, device="cuda").bfloat16()
    call = lambda **kw: ops.bsgemm(a, b, epilogue=ops.EPI_BIAS_RESIDUAL, bias=bias, alpha=0.5, **kw)
    want = call(residual=res)
    assert want.dtype == torch.bfloat16
    assert torch.equal(call(residual=res, out_dtype=torch.float32).bfloat16(), want)
    assert torch.equal(call(residual=res.float(), out_dtype=torch.float32).bfloat16(), want)
