"""CTC top-k at its edges: masked columns, the per-16 format, and the C entry points of the route without logits."""

import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from velox_voice_b200 import ops as m

    return m


def _check(ops, a, b, bias, k):
    logp, ids = ops.bsgemm_topk(a, b, bias, k)
    z = ops.bsgemm(a, b, epilogue=ops.EPI_BIAS, bias=bias, out_dtype=torch.bfloat16)
    ref = torch.log_softmax(z.double(), dim=-1)
    rv = torch.topk(ref, k, dim=-1).values
    assert torch.equal(ref.gather(1, ids), rv)  # the right ids up to ties
    fin = torch.isfinite(rv)
    # log-sum-exp of up to 5,538 fp32 terms, each exponential within 2 ulp; |logits| and |lse| below 16: 2^-20 each
    assert torch.equal(torch.isfinite(logp), fin) and (logp.double() - rv)[fin].abs().max().item() < 4e-5


@pytest.mark.parametrize("N", [64, 264, 5538])
@pytest.mark.parametrize("masked", ["first_piece", "lane", "all_but_16", "tail"])
def test_masked_columns(ops, N, masked):
    """A bias of -inf masks tokens.  The selection kernel reads 8 columns per lane and step of 256: masked are the first
    8, everything that lane 0 reads, all but 16 columns, everything from the second step on."""
    torch.manual_seed(N)
    M, K = 9, 512
    a = ops.quantize(torch.randn(M, K, device="cuda"), "mx32", natural=False)
    b = ops.quantize(0.05 * torch.randn(N, K, device="cuda"), "mx32")
    bias = torch.randn(N, device="cuda")
    col = torch.arange(N, device="cuda")
    mask = {"first_piece": col < 8, "lane": (col % 256) < 8, "all_but_16": (col % (N // 16)) != 3, "tail": col >= 256}[masked]
    bias[mask] = float("-inf")
    _check(ops, a, b, bias, 4)


def test_per_16_format(ops):
    torch.manual_seed(6)
    M, N, K = 130, 5538, 512
    a = ops.quantize(torch.randn(M, K, device="cuda"), "blk16_a")
    b = ops.quantize(0.05 * torch.randn(N, K, device="cuda"), "blk16_b")
    _check(ops, a, b, torch.randn(N, device="cuda"), 5)
