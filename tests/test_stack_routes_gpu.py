"""The stack's native pass against the same layer sequence issued operator by operator, and what a program may change
between passes."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def by_operators(stack, x, pos=None):
    """The pass as separate public calls: bf16 logits and the final residual stream."""
    from velox_voice_b200 import ops

    cfg, fmt, d = stack.cfg, stack.fmt, stack.cfg.d_model
    am = lambda k: stack.amax.get(k)
    nat = fmt == ops.FMT_FP8_1X128
    lnq = lambda k, t: ops.ln_quantize(t, *stack.ln[k], cfg.eps, fmt, amax_t=am(k))
    q = lambda k, t: ops.quantize(t, fmt, natural=nat, amax_t=am(k))
    if pos is not None:
        q("pos", pos)
    a = None
    for i in range(cfg.blocks):
        b = f"b{i}."
        for ff, ln in (("ffm", "ln_ffm"), ("ff", "ln_ff")):
            if a is None or ff == "ff":
                a = lnq(b + ln, x)
            if stack.fuse_ffn:
                h = stack.p[b + ff + ".w1"](a, act="swish", out_fmt=fmt, out_amax=am(b + ff + ".h"))
            else:
                h = q(b + ff + ".h", stack.p[b + ff + ".w1"](a, act="swish"))
            x = stack.p[b + ff + ".w2"](h, residual=x, alpha=0.5)
            if ff == "ffm":
                qkv = stack.p[b + "qkv"](lnq(b + "ln_mha", x))
                x = stack.p[b + "lo"](q(b + "ctx", qkv[:, 2 * d:]), residual=x)
                x = stack.p[b + "pw2"](q(b + "glu", stack.p[b + "pw1"](lnq(b + "ln_conv", x))), residual=x)
        nxt = f"b{i + 1}.ln_ffm" if i + 1 < cfg.blocks else "after"
        y = torch.empty_like(x)
        a = ops.ln2_quantize(x, *stack.ln[b + "ln_final"], *stack.ln[nxt], cfg.eps, fmt, y=y, amax_t=am(nxt))
        x = y
    if a is None:
        a = lnq("after", x)
    return stack.p["ctc"](a), x


def build(fmt="mx32", seed=0, **kw):
    from velox_voice_b200.stack import ConformerLinearStack, StackConfig, make_weights

    cfg = StackConfig(fmt=fmt, **kw)
    w = make_weights(cfg, seed=seed)
    g = torch.Generator().manual_seed(seed)
    for k in w:
        if w[k].dim() == 1:
            w[k] = w[k] + 0.05 * torch.randn(w[k].shape, generator=g)
    stack = ConformerLinearStack(cfg, w)
    if fmt == "nv16":
        x = torch.randn(256, cfg.d_model, generator=g).cuda().bfloat16()
        stack.calibrate(x, x)
    return stack


@pytest.mark.parametrize("fmt,kw", [("mx32", {}), ("nv16", {}), ("fp8_1x128", {}), ("mx32", dict(fuse_ffn=False)), ("nv16", dict(fuse_ffn=False)),
                                    ("mx32", dict(d_model=256, heads=4, ffn=1024, conv_pw=512, vocab=101)),
                                    ("mx32", dict(d_model=384, heads=6, ffn=1536, conv_pw=768, vocab=1000)),
                                    ("nv16", dict(d_model=768, heads=12, ffn=3072, conv_pw=1536, vocab=1000)),
                                    ("mx32", dict(blocks=0))])
def test_native_pass_has_the_bytes_of_the_operators(fmt, kw):
    kw = {"blocks": 2, **kw}
    stack = build(fmt, **kw)
    d = stack.cfg.d_model
    torch.manual_seed(7)
    for T in (1, 130, 777, 5000):
        x = torch.randn(T, d, device="cuda").bfloat16()
        pos = torch.randn(T, d, device="cuda")
        want, hidden = by_operators(stack, x.clone())
        wide = torch.zeros(T, d + 64, device="cuda", dtype=torch.bfloat16)
        wide[:, 32:32 + d] = x
        for xx, pp in ((x.clone(), None), (x.clone(), pos.bfloat16()), (x.clone(), pos), (x.clone(), pos.T.contiguous().T),
                       (wide[:, 32:32 + d], None)):
            got, h = stack.forward(xx, pp, return_hidden=True)
            assert torch.equal(got, want) and torch.equal(h, hidden), T
        buf, src = torch.empty_like(x), x.clone()
        assert torch.equal(stack.forward(buf, pos, source=src), want) and torch.equal(src, x)
        assert torch.equal(stack.forward_ids(x.clone(), pos).long(), want.float().argmax(1))


@pytest.mark.parametrize("fmt", ["mx32", "fp8_1x128"])
def test_no_frames(fmt):
    stack = build(fmt, blocks=2)
    x = torch.empty(0, 512, device="cuda", dtype=torch.bfloat16)
    assert stack.forward(x, x.clone()).shape == (0, stack.cfg.vocab) and stack.forward_ids(x).shape == (0,)


def test_frames_of_the_fused_launches_are_the_callers_to_choose():
    from velox_voice_b200 import ops

    x = torch.randn(5000, 512, device="cuda").bfloat16()
    count = {}
    for least in (None, 1, 5000, 5001, 1 << 30):
        stack = build(blocks=1, **({} if least is None else {"fuse_ln_min_frames": least}))
        ops.reset_launch_count()
        stack.forward_ids(x.clone())
        count[least] = ops.launch_count()
    assert count[1] == count[5000] == count[None] < count[5001] == count[1 << 30]


@pytest.mark.parametrize("frames", [375, 5000])
def test_frames_of_the_fused_launches_may_be_chosen_on_a_built_stack(frames):
    """Assigned later the line holds for passes of every length, as it does when given with the configuration."""
    from velox_voice_b200 import ops

    torch.manual_seed(12)
    x = torch.randn(frames, 512, device="cuda").bfloat16()
    stack = build(blocks=1)
    want = stack.forward(x.clone())
    for least in (0, frames, frames + 1):
        count = []
        for given in (build(blocks=1, fuse_ln_min_frames=least), stack):
            given.fuse_ln_min_frames = least
            ops.reset_launch_count()
            assert torch.equal(given.forward(x.clone()), want)
            count.append(ops.launch_count())
        assert count[0] == count[1] == (14 if least > frames else 10)


def test_what_a_program_replaces_takes_effect():
    """Layers, their weights and biases, LayerNorm parameters and calibrated maxima may be replaced between passes."""
    torch.manual_seed(8)
    x = torch.randn(200, 512, device="cuda").bfloat16()
    other = build(seed=1, blocks=2)
    stack = build(blocks=2)

    def check():
        want, _ = by_operators(stack, x.clone())
        assert torch.equal(stack.forward(x.clone()), want)
        return want

    seen = [check()]
    stack.p["b1.pw2"] = other.p["b1.pw2"]
    seen.append(check())
    stack.p["b0.qkv"].q = other.p["b0.qkv"].q
    seen.append(check())
    stack.p["ctc"].bias = other.p["ctc"].bias + 1.0
    seen.append(check())
    stack.ln["b0.ln_conv"] = (1.5 * stack.ln["b0.ln_conv"][0], stack.ln["b0.ln_conv"][1])
    seen.append(check())
    stack.ln["b1.ln_ff"] = tuple(t.bfloat16() for t in stack.ln["b1.ln_ff"])
    seen.append(check())
    stack.ln["b1.ln_ff"][0].mul_(2.0)  # in place, where the kernels read a converted copy
    seen.append(check())
    stack.ln["b1.ln_ff"] = (torch.rand(1024, device="cuda")[::2], stack.ln["b1.ln_ff"][1])
    seen.append(check())
    stack.ln["b1.ln_ff"][0].add_(0.5)
    seen.append(check())
    stack.cfg.eps = 1e-2
    seen.append(check())
    stack.fuse_ffn = False
    check()
    assert all(not torch.equal(a, b) for a, b in zip(seen, seen[1:]))
    stack = build("nv16", blocks=2)
    first = check()
    stack.amax["b0.ln_mha"] = 1.3 * stack.amax["b0.ln_mha"]
    assert not torch.equal(check(), first)


def test_new_tensors_and_storage_of_a_layer_take_effect():
    """The fields of a layer's packed weight may be assigned, and a tensor may be given other storage: the pointers of the plan
    would lead to the former one."""
    torch.manual_seed(11)
    x = torch.randn(200, 512, device="cuda").bfloat16()
    for fmt in ("mx32", "nv16", "fp8_1x128"):
        stack, other = build(fmt, blocks=2), build(fmt, seed=1, blocks=2)
        scales = "scales" if fmt == "fp8_1x128" else "sf"

        def changed(before):
            want, _ = by_operators(stack, x.clone())
            assert torch.equal(stack.forward(x.clone()), want) and not torch.equal(want, before)
            return want

        last = stack.forward(x.clone())
        a, b = stack.p["b0.lo"].q, other.p["b0.lo"].q
        a.codes = b.codes
        last = changed(last)
        setattr(a, scales, getattr(b, scales).roll(1, 0).contiguous())
        last = changed(last)
        stack.p["b1.pw1"].q.codes.data = other.p["b1.pw1"].q.codes.clone()
        last = changed(last)
        stack.p["b1.qkv"].bias.data = stack.p["b1.qkv"].bias + 1.0
        last = changed(last)
        stack.ln["after"][0].data = 2.0 * stack.ln["after"][0]
        last = changed(last)
        if fmt == "nv16":
            a.amax = 2.0 * a.amax
            last = changed(last)
            a.amax.data = 2.0 * a.amax
            changed(last)


def test_widths_come_from_the_weights():
    """The configuration's ffn, conv_pw and vocab describe a model; a pass runs the layers as they are.  What does not fit the
    layer before it is refused."""
    from velox_voice_b200.stack import ConformerLinearStack, StackConfig, make_weights

    torch.manual_seed(9)
    small = StackConfig(blocks=2, ffn=1024, conv_pw=512, vocab=999)
    w = make_weights(small, seed=4)
    stack = ConformerLinearStack(StackConfig(blocks=2), w)
    x = torch.randn(140, 512, device="cuda").bfloat16()
    want, _ = by_operators(stack, x.clone())
    assert want.shape[1] == 999 and torch.equal(stack.forward(x.clone()), want)
    stack.p["b0.ff.w1"] = build(blocks=1).p["b0.ff.w1"]  # 2,048 outputs in front of 1,024 inputs
    with pytest.raises(ValueError):
        stack.forward(x.clone())


@pytest.mark.parametrize("fmt", ["mx32", "nv16", "fp8_1x128"])
def test_a_plan_points_into_the_layers(fmt):
    """Making the plan of a pass runs nothing on the device and makes no copies: it happens in the first pass, whose stream
    or graph capture later passes need not have waited for."""
    stack = build(fmt, blocks=3)
    torch.cuda.synchronize()
    before = torch.cuda.memory_stats()["allocation.all.allocated"]
    stack._host_plan()
    assert torch.cuda.memory_stats()["allocation.all.allocated"] == before
    whole = stack._positions
    assert (whole is None) == (fmt == "nv16")
    if whole is None:
        return
    for i in range(3):
        q = stack.p[f"b{i}.lp"].q
        for name in ("codes", "scales", "sf"):
            part, t = getattr(q, name), getattr(whole, name)
            assert (part is None) == (t is None)
            assert t is None or part.data_ptr() == t[i * t.shape[0] // 3].data_ptr()
    x = torch.zeros(8, 512, device="cuda", dtype=torch.bfloat16)

    def launches():
        ops.reset_launch_count()
        stack.forward_ids(x.clone(), x)
        return ops.launch_count()

    from velox_voice_b200 import ops

    together = launches()
    stack.p["b1.lp"].q.codes = stack.p["b1.lp"].q.codes.clone()
    assert launches() == together + 2  # a launch per block


def test_first_pass_on_another_stream_and_in_a_capture():
    torch.manual_seed(10)
    x, pos = (torch.randn(300, 512, device="cuda").bfloat16() for _ in range(2))
    want, _ = by_operators(build(blocks=2), x.clone())
    stack = build(blocks=2)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    got = []
    for s in streams:
        with torch.cuda.stream(s):
            got.append(stack.forward(x.clone(), pos))
    torch.cuda.synchronize()
    assert all(torch.equal(g, want) for g in got)
    stack = build(blocks=2)
    stack.forward(x.clone())  # (one-time module loading is not to be captured; the plan is)
    stack._plan = None
    buf, graph = x.clone(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        out = stack.forward(buf, pos)
    assert torch.equal(stack.forward(x.clone(), pos), want)  # before any replay
    buf.copy_(x)
    graph.replay()
    assert torch.equal(out, want)


@pytest.mark.parametrize("fmt,frames", [("mx32", 375), ("mx32", 4200), ("mx32", 4500), ("mx32", 5000), ("nv16", 375)])
def test_the_launches_of_the_benchmark_are_those_of_a_pass(fmt, frames):
    from velox_voice_b200 import opbench, ops

    stack = build(fmt, blocks=2)
    x = torch.randn(frames, 512, device="cuda").bfloat16()
    cases = opbench.op_breakdown(stack, frames, fmt)
    ops.reset_launch_count()
    stack.forward_ids(x.clone(), x)
    # the entry for all blocks holds the head and, as the head's own entry, the launch that turns keys into ids
    whole = any(n.startswith("all blocks") for n, *_ in cases)
    assert whole == (fmt == "mx32" and frames <= stack.one_launch_frames)
    assert sum(c for _, c, *_ in cases) + (2 if whole else 1) == ops.launch_count()
