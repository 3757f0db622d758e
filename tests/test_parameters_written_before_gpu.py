"""Biases, LayerNorm parameters and filterbanks that the launch before wrote: a library GEMM triggers the launch behind it early, and what
that launch reads is what the GEMM wrote, in eager calls and on a captured chain."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def stale(rows, cols, call):
    """How many of the results of `call(parameters f32 [rows, cols])` right behind the GEMM that writes the parameters differ from
    those behind a synchronisation, for eight sets of parameters."""
    from velox_voice_b200 import _lib, ops

    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda")
    par = torch.zeros(rows, cols, device="cuda")
    w = ops.quantize(randn(cols, 2048), "mx32")
    acts = [ops.quantize(randn(rows, 2048), "mx32") for _ in range(8)]
    want = []
    for a in acts:
        ops.bsgemm(a, w, out=par)
        torch.cuda.synchronize()
        want.append(call(par))
    assert not torch.equal(want[0], want[1])

    def chain():
        got = []
        for a in acts:
            ops.bsgemm(a, w, out=par)
            got.append(call(par))
        return got

    bad = 0
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = chain()
    for _ in range(10):
        bad += sum(not torch.equal(x, y) for x, y in zip(chain(), want))
        graph.replay()
        bad += sum(not torch.equal(x, y) for x, y in zip(captured, want))
    assert _lib.device_status() == 0
    return bad


@pytest.mark.parametrize("fmt,K", [("mx32", 512), ("nv16", 512), ("fp8_1x128", 512), ("mx32", 256), ("mx32", 1024), ("nv16", 2048), ("rowscale", 512)])
@pytest.mark.parametrize("M", [100, 4000])
def test_layernorm_quantizers(fmt, K, M):
    from velox_voice_b200 import ops

    x = torch.randn(M, K, device="cuda").bfloat16()
    one = torch.ones(K, device="cuda")
    am = dict(amax_t=torch.tensor([6.0], device="cuda")) if fmt == "nv16" else {}
    assert stale(1, K, lambda p: ops.ln_quantize(x, p[0], one, 1e-5, fmt, **am).codes) == 0
    assert stale(1, K, lambda p: ops.ln_quantize(x, one, p[0], 1e-5, fmt, **am).codes) == 0
    if fmt == "mx32":
        assert stale(2, K, lambda p: ops.ln2_quantize(x, one, p[0], p[1], one, 1e-5, fmt, y=torch.empty_like(x)).codes) == 0
        assert stale(2, K, lambda p: ops.layernorm(x, p[0], p[1], 1e-5)) == 0


@pytest.mark.parametrize("K", [512, 2048])
@pytest.mark.parametrize("M", [100, 10000])
def test_residual_layernorm_gemm(M, K):
    from velox_voice_b200 import ops
    from velox_voice_b200.linear import PackedLinear

    lin = PackedLinear(0.05 * torch.randn(512, K, device="cuda"), torch.zeros(512, device="cuda"), "mx32")
    a = ops.quantize(torch.randn(M, K, device="cuda").bfloat16(), "mx32")
    res, one = torch.randn(M, 512, device="cuda").bfloat16(), torch.ones(512, device="cuda")

    def call(bias=one, gamma=one, beta=one, **two):
        lin.bias = bias
        return lin.residual_ln(a, residual=res, gamma=gamma, beta=beta, eps=1e-5, alpha=1.0, **two)[1].codes

    assert stale(1, 512, lambda p: call(bias=p[0])) == 0
    assert stale(2, 512, lambda p: call(gamma=p[0], beta=p[1])) == 0
    assert stale(2, 512, lambda p: call(gamma2=p[0], beta2=p[1])) == 0


@pytest.mark.parametrize("M,F", [(80, 257), (3, 257), (80, 256), (130, 257)])  # one copy, its remainder of three, word by word, the other kernel
def test_filterbank(M, F):
    from velox_voice_b200 import ops

    spec = torch.randn(1000, F, dtype=torch.complex64, device="cuda")
    zero, one = torch.zeros(M, device="cuda"), torch.ones(M, device="cuda")
    assert stale(M, F, lambda p: ops.power_mel_log(spec, p, zero, one)) == 0
    bank = torch.linspace(0.0, 1.0, M * F, device="cuda").view(M, F)
    assert stale(2, M, lambda p: ops.power_mel_log(spec, bank, p[0], p[1])) == 0


@pytest.mark.parametrize("M", [1, 16, 300])
def test_bias_of_the_per_row_lane(M):
    from velox_voice_b200 import ops

    x = torch.randn(M, 512, device="cuda")
    wq, ws = ops.per_row_col_quantize(0.02 * torch.randn(2048, 512, device="cuda"))
    assert stale(1, 2048, lambda p: ops.rowscale_linear(x, wq, ws, p[0])) == 0
