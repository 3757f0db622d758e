"""A per-row-scaled linear on few rows in one launch (``vx_rowscale.cu``) against the quantizer and the GEMM as two calls,
bit for bit, around the edges of its row tiles, column groups, K chunks and of its range."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 8, 128), (1, 1, 32768), (3, 512, 9728), (4, 512, 9728), (15, 2048, 512), (16, 2048, 512), (17, 5538, 512),
                                   (31, 7, 1024), (32, 200, 1024), (33, 1536, 512), (63, 9, 384), (64, 2048, 512), (65, 2048, 512),
                                   (16, 512, 2048), (17, 512, 2048), (5, 300, 96), (64, 5538, 256)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_equals_the_two_calls(M, N, K, dtype):
    from velox_voice_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(M * N + K)
    x = (torch.randn(M, K, generator=g, device="cuda") * torch.logspace(-2, 2, M, device="cuda")[:, None]).to(dtype)
    x[M // 2, ::3] = 0
    x[0, 0] = -1e-30
    wq, ws = ops.quantize_w(0.02 * torch.randn(N, K, generator=g, device="cuda"))
    bias = torch.randn(N, generator=g, device="cuda")
    a, b = ops.quantize(x, "rowscale", sf=False), ops._as_quantized_rowscale(wq, ws)
    assert torch.equal(ops.rowscale_linear(x, wq, ws, bias), ops.bsgemm(a, b, epilogue=ops.EPI_BIAS, bias=bias, out_dtype=torch.float32))
    assert torch.equal(ops.rowscale_linear(x, wq, ws), ops.bsgemm(a, b, out_dtype=torch.float32))
