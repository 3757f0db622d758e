"""The native host path (csrc/vx_host.cpp) against the Python route of the same operators: equal bytes for every form
of argument that both take, the same refusals, and the module and stack behaviour that callers rely on."""

import pytest
import torch

pytestmark = pytest.mark.gpu

FMTS = ("rowscale", "mx32", "nv16", "fp8_1x128")


@pytest.fixture(scope="module")
def ops():
    from velox_voice_b200 import ops as m

    m._host()
    return m


class _NoHost:
    """Every operator answers None, as the native functions do for arguments they leave to the Python route."""

    def __getattr__(self, name):
        return lambda *a: None


def both_routes(ops, monkeypatch, call):
    """(result or exception type) of the call on the native and on the Python route."""
    out = []
    for host in (ops._native, _NoHost()):
        with monkeypatch.context() as m:
            m.setattr(ops, "_native", host)
            try:
                out.append(call())
            except Exception as e:
                out.append(type(e))
    return out


def same(a, b):
    if isinstance(a, type) or isinstance(b, type):
        return a is b
    if isinstance(a, (tuple, list)):
        return len(a) == len(b) and all(same(x, y) for x, y in zip(a, b))
    if isinstance(a, torch.Tensor):
        return a.dtype == b.dtype and a.shape == b.shape and torch.equal(a.contiguous().view(torch.uint8), b.contiguous().view(torch.uint8))
    if a is None or b is None:
        return a is b
    return (a.fmt, a.rows, a.k) == (b.fmt, b.rows, b.k) and all(same(getattr(a, f), getattr(b, f)) for f in ("codes", "scales", "sf", "amax"))


def views(x):
    """One matrix in the layouts callers have it in: contiguous, rows of a wider buffer, every second row, transposed storage,
    16-byte offset inside a buffer, and one element off (rows no longer 16-byte aligned)."""
    R, C = x.shape
    wide = torch.zeros(R, C + 64, dtype=x.dtype, device=x.device)
    wide[:, 32:32 + C] = x
    gaps = torch.zeros(2 * R, C, dtype=x.dtype, device=x.device)
    gaps[::2] = x
    flat = torch.zeros(R * C + 64, dtype=x.dtype, device=x.device)
    off = flat[8:8 + R * C].view(R, C).copy_(x)
    odd = torch.zeros(R * C + 64, dtype=x.dtype, device=x.device)[1:1 + R * C].view(R, C).copy_(x)
    return {"dense": x, "wide": wide[:, 32:32 + C], "gaps": gaps[::2], "columns": x.T.contiguous().T, "offset": off, "odd": odd,
            "half": x.half()}


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("fmt", FMTS)
def test_quantizers_agree_on_both_routes(ops, monkeypatch, fmt, dtype):
    torch.manual_seed(1)
    x = torch.randn(130, 512, device="cuda").to(dtype)
    g, b = 1 + 0.1 * torch.randn(512, device="cuda"), 0.1 * torch.randn(512, device="cuda")
    am = torch.tensor([5.0], device="cuda") if fmt == "nv16" else None
    for name, v in views(x).items():
        for nat in (True, False, 1, 0):
            r = both_routes(ops, monkeypatch, lambda: ops.quantize(v, fmt, natural=nat, amax_t=am))
            assert same(*r), (name, nat)
        for gg, bb in ((g, b), (g.bfloat16(), b.bfloat16()), (g.repeat_interleave(2)[::2], b)):
            r = both_routes(ops, monkeypatch, lambda: ops.ln_quantize(v, gg, bb, 1e-5, fmt, sf=1, amax_t=am))
            assert same(*r), (name, gg.dtype)
    for rows in (0, 1):
        r = both_routes(ops, monkeypatch, lambda: ops.quantize(x[:rows], fmt, amax_t=am))
        assert same(*r), rows
    if fmt == "nv16":
        assert same(*both_routes(ops, monkeypatch, lambda: ops.quantize(x, fmt)))  # measures the maximum itself
    for bad in (x[0], x.cpu(), x.reshape(13, 10, 512)):
        r = both_routes(ops, monkeypatch, lambda: ops.quantize(bad, fmt, amax_t=am))
        assert isinstance(r[0], type) and r[0] is r[1]


@pytest.mark.parametrize("fmt", FMTS)
def test_gemms_agree_on_both_routes(ops, monkeypatch, fmt):
    from velox_voice_b200.ops import EPI_BIAS, EPI_BIAS_RESIDUAL, EPI_BIAS_SWISH, EPI_NONE

    torch.manual_seed(2)
    M, N, K = 130, 512, 512
    a = ops.quantize(torch.randn(M, K, device="cuda"), fmt)
    w = ops.quantize(0.05 * torch.randn(N, K, device="cuda"), fmt)
    bias = torch.randn(N, device="cuda")
    out = torch.empty(M, N + 8, device="cuda")[:, :N]
    for kw in (dict(), dict(epilogue=EPI_BIAS, bias=bias), dict(epilogue=EPI_BIAS_SWISH, bias=bias, out_dtype=torch.float32),
               dict(epilogue=EPI_BIAS, bias=bias[:100]), dict(epilogue=EPI_BIAS, bias=bias.double()), dict(out_dtype=torch.float16),
               dict(epilogue=EPI_BIAS, bias=bias, out=out), dict(out=out.T), dict(epilogue=EPI_BIAS_RESIDUAL, bias=bias)):
        r = both_routes(ops, monkeypatch, lambda: ops.bsgemm(a, w, **kw))
        assert same(*r), kw.keys()
    for name, res in views(torch.randn(M, N, device="cuda").bfloat16()).items():
        for r32 in (res, res.float() if name == "dense" else res):
            r = both_routes(ops, monkeypatch, lambda: ops.bsgemm(a, w, epilogue=EPI_BIAS_RESIDUAL, bias=bias, residual=r32, alpha=0.5))
            assert same(*r), name
    if fmt in ("mx32", "nv16"):
        am = torch.tensor([8.0], device="cuda") if fmt == "nv16" else None
        r = both_routes(ops, monkeypatch, lambda: ops.bsgemm(a, w, epilogue=EPI_BIAS_SWISH, bias=bias, out_fmt=fmt, out_amax=am, out_natural=1))
        assert same(*r)
    if fmt == "mx32":
        g, b = torch.ones(N, device="cuda"), torch.zeros(N, device="cuda")
        res = torch.randn(M, N, device="cuda").bfloat16()
        for gg in (g, g.bfloat16()):
            r = both_routes(ops, monkeypatch, lambda: ops.bsgemm_residual_ln(a, w, bias=bias, residual=res, gamma=gg, beta=b, eps=1e-5))
            assert same(*r)
    assert same(*both_routes(ops, monkeypatch, lambda: ops.bsgemm(a, ops.quantize(torch.randn(N, 256, device="cuda"), fmt), epilogue=EPI_NONE)))


def test_remaining_operators_agree_on_both_routes(ops, monkeypatch):
    torch.manual_seed(3)
    wq, ws = ops.per_row_col_quantize(0.05 * torch.randn(200, 512, device="cuda"))
    bias = torch.randn(200, device="cuda")
    for rows in (1, 5, 64, 130):
        for name, x in views(torch.randn(rows, 512, device="cuda")).items():
            for b in (bias, None, bias.bfloat16(), bias.repeat_interleave(2)[::2]):
                r = both_routes(ops, monkeypatch, lambda: ops.rowscale_linear(x, wq, ws, b))
                assert same(*r), (rows, name)
    aq, asc = ops.mxfp4_block_quantize(torch.randn(130, 512, device="cuda").bfloat16(), "A")
    bq, bsc = ops.mxfp4_block_quantize(torch.randn(200, 512, device="cuda").bfloat16(), "B")
    for sa in (asc, asc.T.contiguous().T):
        assert same(*both_routes(ops, monkeypatch, lambda: ops.dgx_mxfp4_blkscale_gemm(aq, bq, sa, bsc)))
    spec = torch.randn(130, 257, dtype=torch.complex64, device="cuda")
    mel, mean, istd = torch.rand(80, 257, device="cuda"), torch.randn(80, device="cuda"), torch.rand(80, device="cuda")
    for s in (spec, spec[:64], spec[:63], spec.conj(), spec.to(torch.complex128), spec.T.contiguous().T, spec[1:]):
        for m in (mel, mel.T.contiguous().T, mel.double()):
            r = both_routes(ops, monkeypatch, lambda: ops.power_mel_log(s, m, mean, istd))
            assert same(*r), (s.shape, s.dtype)
    h, T = 2, 130
    qkv = [torch.randn(h, T, 128, device="cuda").bfloat16() for _ in range(3)]
    for kv in (None, 0, 65, T, T + 1):
        assert same(*both_routes(ops, monkeypatch, lambda: ops.relpos_attention(*qkv, kv)))
    assert same(*both_routes(ops, monkeypatch, lambda: ops.relpos_attention(qkv[0], qkv[1].transpose(0, 1).contiguous().transpose(0, 1), qkv[2])))


def test_dense_linear_bias_need_not_be_a_parameter():
    """Pruning and parametrization turn `bias` into a plain attribute or a property of the module."""
    from torch.nn.utils import parametrize

    from velox_voice_b200.linear import DenseLinear

    torch.manual_seed(5)
    w, b = torch.randn(256, 128), torch.randn(256)
    x = torch.randn(20, 128, device="cuda")

    def make():
        lin = DenseLinear(w, b).cuda().requires_grad_(False)
        lin.precision = "mxfp4"
        return lin

    want = make()(x)
    lin = make()
    bias = lin.bias.detach()
    del lin.bias
    lin.bias = bias
    assert torch.equal(lin(x), want)
    lin = make()
    parametrize.register_parametrization(lin, "bias", torch.nn.Identity())
    assert torch.equal(lin(x), want)


def test_rowscale_linear_takes_matrices_only(ops):
    wq, ws = ops.per_row_col_quantize(torch.randn(64, 128, device="cuda"))
    for shape in ((128,), (2, 3, 128)):
        with pytest.raises(ValueError):
            ops.rowscale_linear(torch.randn(*shape, device="cuda"), wq, ws)


def test_fold_pack_takes_unaligned_fp32_biases(ops):
    """fp32 positional biases at any address: a slice of a parameter that does not start on 16 bytes."""
    torch.manual_seed(4)
    h, dk, M = 8, 64, 70
    a = ops.quantize(torch.randn(M, 512, device="cuda"), "mx32")
    w = ops.quantize(0.05 * torch.randn(3 * h * dk, 512, device="cuda"), "mx32")
    u, v = torch.randn(h, dk, device="cuda"), torch.randn(h, dk, device="cuda")
    buf = torch.empty(2 * h * dk + 3, device="cuda")
    uo, vo = buf[1:1 + h * dk].view(h, dk).copy_(u), buf[3 + h * dk:].view(h, dk).copy_(v)
    for uu, vv in ((uo, v), (u, vo)):
        got = ops.bsgemm_qkv_pack(a, w, None, uu, vv, 0.125)
        want = ops.bsgemm_qkv_pack(a, w, None, u, v, 0.125)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1][..., :dk], want[1][..., :dk]) and torch.equal(got[2], want[2])


def test_host_calls_release_the_interpreter():
    """A forward pass that blocks in its launches (the stream's queue is full) lets other Python threads run."""
    import threading
    import time

    from velox_voice_b200.stack import ConformerLinearStack, StackConfig, make_weights

    cfg = StackConfig(blocks=2)
    stack = ConformerLinearStack(cfg, make_weights(cfg))
    x, pos = torch.randn(128, 512, device="cuda").bfloat16(), torch.randn(128, 512, device="cuda").bfloat16()
    stack.forward_ids(x.clone(), pos)
    torch.cuda.synchronize()
    ticks, stop = [], threading.Event()

    def tick():
        while not stop.is_set():
            ticks.append(time.perf_counter())
            time.sleep(0.002)

    t = threading.Thread(target=tick)
    t.start()
    try:
        torch.cuda._sleep(1_500_000_000)  # about 0.8 s of an occupied stream
        t0 = time.perf_counter()
        while time.perf_counter() - t0 < 0.25:  # fill the queue until a call blocks
            t1 = time.perf_counter()
            for _ in range(20):
                stack.forward_ids(x, pos)
            if time.perf_counter() - t1 > 0.2:
                break
    finally:
        end = time.perf_counter()
        stop.set()
        t.join()
    torch.cuda.synchronize()
    seen = [v for v in ticks if t0 <= v <= end]
    assert end - t0 > 0.2, "the queue never filled"
    gaps = [b - a for a, b in zip([t0] + seen, seen + [end])]
    assert max(gaps) < 0.1, f"no other thread ran for {max(gaps):.3f} s of {end - t0:.3f} s"
