"""What a user of this library has it do, as cases that can be timed: the reference's drop-in linears, the
encoder's linears, modules and whole stack in the formats they run in, the CTC tail and the front-end's
filterbank, each through the public entry points and over the sizes they meet.

Sizes: encoder frames are 40 ms.  A streaming chunk has 16 of them, an utterance tens to thousands, a
span of long audio at most 3,750, a batch of sixteen one-minute utterances 24,000 and an hour of audio
about 90,000 (360,000 filterbank frames of 10 ms)."""

import math

import torch

from velox_voice_b200 import ops
from velox_voice_b200.linear import DenseLinear, PackedLinear
from velox_voice_b200.stack import ConformerLinearStack, StackConfig

D, HEADS, FFN, VOCAB = 512, 8, 2048, 5538
BITS = {"mx32": 4 + 8 / 32, "nv16": 4 + 8 / 16, "fp8_1x128": 8 + 32 / 128, "rowscale": 4, "blk16": 4 + 8 / 16}
# (outputs, inputs) of the model's linears: feed-forward up / down, attention, CTC head, subsampling projection
LINEARS = ((2048, 512), (512, 2048), (512, 512), (1536, 512), (5538, 512), (512, 9728))


def listed():
    return [
        # one streaming chunk through one linear of the reference's FP4 lane: launches and host time only
        {"name": "dense_chunk", "kind": "dense", "rows": 16, "n": 2048, "k": 512, "dtype": "float32"},
        # the same lane on a full span of long audio
        {"name": "dense_span", "kind": "dense", "rows": 3750, "n": 512, "k": 2048, "dtype": "float32"},
        # per-16 block-scaled lane of the reference: both sides quantized, fp32 product
        {"name": "blkscale_mid", "kind": "blkscale", "rows": 1022, "n": 512, "k": 1024},
        # convolution module's pointwise GLU on an ordinary utterance: quantize + GEMM
        {"name": "glu_utterance", "kind": "linear", "op": "glu", "fmt": "mx32", "frames": 1537},
        # fused q|k|v projection in FP8 for an hour of audio: quantize + GEMM
        {"name": "qkv_fp8_hour", "kind": "linear", "op": "qkv", "fmt": "fp8_1x128", "frames": 90000},
        # macaron feed-forward in NVFP4 for an hour of audio: LayerNorm, up, Swish, down, residual
        {"name": "ffn_nv16_hour", "kind": "ffn", "fmt": "nv16", "frames": 90000},
        # attention module of one block on a full span: LayerNorm, q|k|v, positions, attention, output projection
        {"name": "attention_span", "kind": "attention", "frames": 3750},
        # what the prefix beam search takes: the five best log-probabilities of every frame of a span
        {"name": "topk_span", "kind": "topk", "frames": 3750, "k": 5},
        # front-end's filterbank for an hour of audio
        {"name": "mel_hour", "kind": "mel", "frames": 360000, "bins": 257, "mels": 80},
        # greedy transcription of a short utterance whose length nobody knew before: launches and host time
        {"name": "stack_utterance", "kind": "stack", "mode": "eager_ids", "frames": 375},
        # a batch of sixteen one-minute utterances, logits wanted
        {"name": "stack_batch_logits", "kind": "stack", "mode": "logits", "frames": 24000},
        # an hour of audio, greedy, on the captured stack
        {"name": "stack_hour", "kind": "stack", "mode": "graph_ids", "frames": 89999},
    ]


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("dense", "dense", "blkscale", "linear", "linear", "ffn", "attention", "topk", "mel",
                       "eager_ids", "logits", "graph_ids"))
    if kind == "dense":
        n, k = rng.choice(LINEARS)
        return {"kind": kind, "rows": _log_size(rng, 1, 3750), "n": n, "k": k,
                "dtype": rng.choice(("float32", "bfloat16"))}
    if kind == "blkscale":
        n, k = rng.choice(((200, 512), (256, 512), (512, 1024), (512, 2048), (2048, 2048)))
        return {"kind": kind, "rows": 2 * _log_size(rng, 32, 1900), "n": n, "k": k}
    if kind == "linear":
        return {"kind": kind, "op": rng.choice(("glu", "qkv")), "fmt": rng.choice(("mx32", "nv16", "fp8_1x128")),
                "frames": _log_size(rng, 64, 90000)}
    if kind == "ffn":
        return {"kind": kind, "fmt": rng.choice(("mx32", "nv16")), "frames": _log_size(rng, 256, 90000)}
    if kind == "attention":
        return {"kind": kind, "frames": _log_size(rng, 100, 3750)}
    if kind == "topk":
        return {"kind": kind, "frames": _log_size(rng, 50, 15000), "k": rng.choice((1, 5, 8, 10))}
    if kind == "mel":
        return {"kind": kind, "frames": _log_size(rng, 200, 360000), "bins": 257, "mels": 80}
    lo, hi = {"eager_ids": (16, 6000), "logits": (375, 24000), "graph_ids": (375, 89999)}[kind]
    return {"kind": "stack", "mode": kind, "frames": _log_size(rng, lo, hi)}


def _stack_weights(cfg, randn):
    """Weights of the stack under the names it takes: N(0, 0.02), small biases, LayerNorm near the identity."""
    d, f = cfg.d_model, cfg.ffn
    w = {}

    def linear(name, n, k, b=True):
        dot = name.rfind(".w")
        w[name] = 0.02 * randn(n, k)
        if b:
            w[name[:dot] + ".b" + name[dot + 2:]] = 0.02 * randn(n)

    def norm(name):
        w[name + ".g"], w[name + ".b"] = 1.0 + 0.05 * randn(d), 0.05 * randn(d)

    for i in range(cfg.blocks):
        p = f"b{i}."
        for ff in ("ffm", "ff"):
            linear(p + ff + ".w1", f, d)
            linear(p + ff + ".w2", d, f)
        linear(p + "qkv.w", 3 * d, d)
        linear(p + "lo.w", d, d)
        linear(p + "lp.w", d, d, b=False)
        linear(p + "pw1.w", cfg.conv_pw, d)
        linear(p + "pw2.w", d, cfg.conv_pw // 2)
        for n in ("ln_ffm", "ln_mha", "ln_conv", "ln_ff", "ln_final"):
            norm(p + n)
    norm("after")
    linear("ctc.w", cfg.vocab, d)
    return w


def _filterbank(mels, bins, device):
    """Triangular filters, evenly spaced on the mel scale up to 8 kHz: f32 [mels, bins]."""
    hz = torch.linspace(0.0, 8000.0, bins, dtype=torch.float64, device=device)
    mel = 1127.0 * torch.log1p(hz / 700.0)
    edges = torch.linspace(float(mel[1]) / 2, float(mel[-1]), mels + 2, dtype=torch.float64, device=device)
    lo, mid, hi = edges[:-2, None], edges[1:-1, None], edges[2:, None]
    return torch.minimum((mel - lo) / (mid - lo), (hi - mel) / (hi - mid)).clamp_min(0.0).float()


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev).manual_seed(seed)

    def randn(*shape):
        return torch.randn(*shape, generator=g, device=dev)

    kind = case["kind"]
    s = {"case": case}
    if kind == "dense":
        # the drop-in module as the reference's loader leaves it: weight quantized once, activations fp32 or bf16
        lin = DenseLinear(0.02 * randn(case["n"], case["k"]), 0.02 * randn(case["n"])).to(dev).requires_grad_(False)
        lin.precision = "mxfp4"
        lin._prequantize_weight("mxfp4")
        s.update(lin=lin, x=randn(case["rows"], case["k"]).to(getattr(torch, case["dtype"])))
    elif kind == "blkscale":
        wq, ws = ops.mxfp4_block_quantize((0.02 * randn(case["n"], case["k"])).bfloat16(), mode="B")
        s.update(x=randn(case["rows"], case["k"]).bfloat16(), wq=wq, ws=ws)
    elif kind == "linear":
        glu = case["op"] == "glu"
        n = 2 * D if glu else 3 * D
        lin = PackedLinear(0.03 * randn(n, D), 0.02 * randn(n), case["fmt"], glu=glu)
        s.update(lin=lin, x=torch.nn.functional.layer_norm(randn(case["frames"], D), (D,)).bfloat16())
    elif kind == "ffn":
        # NV16 tensor scales are calibrated before serving: LayerNorm outputs and the Swish intermediate
        nv = case["fmt"] == "nv16"
        s.update(x=randn(case["frames"], D).bfloat16(), g=1.0 + 0.05 * randn(D), b=0.05 * randn(D),
                 up=PackedLinear(0.02 * randn(FFN, D), 0.02 * randn(FFN), case["fmt"]),
                 down=PackedLinear(0.02 * randn(D, FFN), 0.02 * randn(D), case["fmt"]),
                 am_x=torch.tensor([6.0], device=dev) if nv else None, am_h=torch.tensor([4.0], device=dev) if nv else None)
    elif kind == "attention":
        dk = D // HEADS
        s.update(x=randn(case["frames"], D).bfloat16(), pos=randn(case["frames"], D).bfloat16(),
                 g=1.0 + 0.05 * randn(D), b=0.05 * randn(D),
                 qkv=PackedLinear(0.05 * randn(3 * D, D), 0.02 * randn(3 * D), "mx32"),
                 lp=PackedLinear(0.05 * randn(D, D), None, "mx32"), lo=PackedLinear(0.02 * randn(D, D), 0.02 * randn(D), "mx32"),
                 u=0.1 * randn(HEADS, dk), v=0.1 * randn(HEADS, dk), scale=dk ** -0.5)
    elif kind == "topk":
        s.update(head=PackedLinear(0.05 * randn(VOCAB, D), 0.02 * randn(VOCAB), "mx32"),
                 x=randn(case["frames"], D).bfloat16(), g=1.0 + 0.05 * randn(D), b=0.05 * randn(D))
    elif kind == "mel":
        # half spectra of audio-like loudness with a falling spectral slope
        slope = torch.logspace(1.0, -1.0, case["bins"], device=dev)
        spec = torch.randn(case["frames"], case["bins"], dtype=torch.complex64, generator=g, device=dev) * slope
        s.update(spec=spec, mel=_filterbank(case["mels"], case["bins"], dev), mean=randn(case["mels"]),
                 istd=0.5 + torch.rand(case["mels"], generator=g, device=dev))
    elif kind == "stack":
        cfg = StackConfig(fmt="mx32")
        stack = ConformerLinearStack(cfg, _stack_weights(cfg, randn), device=dev)
        x, pos = randn(case["frames"], D).bfloat16(), randn(case["frames"], D).bfloat16()
        if case["mode"] == "graph_ids":
            comp = stack.compile(case["frames"])
            comp.x_in.copy_(x)
            comp.pos.copy_(pos)
            s.update(comp=comp)
        else:
            s.update(stack=stack, x=x, pos=pos)
    else:
        raise ValueError(kind)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "dense":
        return s["lin"](s["x"])
    if kind == "blkscale":
        xq, xs = ops.mxfp4_block_quantize(s["x"], mode="A")
        return ops.mxfp4_gemm(xq, s["wq"], xs, s["ws"])
    if kind == "linear":
        return s["lin"](ops.quantize(s["x"], case["fmt"]))
    if kind == "ffn":
        q = ops.ln_quantize(s["x"], s["g"], s["b"], 1e-5, case["fmt"], amax_t=s["am_x"])
        h = s["up"](q, act="swish", out_fmt=case["fmt"], out_amax=s["am_h"])
        return s["down"](h, residual=s["x"], alpha=0.5)
    if kind == "attention":
        q = ops.ln_quantize(s["x"], s["g"], s["b"], 1e-5, "mx32")
        packed = ops.bsgemm_qkv_pack(q, s["qkv"].q, s["qkv"].bias, s["u"], s["v"], s["scale"])
        ops.bsgemm_heads(ops.quantize(s["pos"], "mx32"), s["lp"].q, None, packed[1], col_off=D // HEADS)
        ctx = ops.relpos_attention(packed[0], packed[1], packed[2])
        return s["lo"](ops.quantize(ctx, "mx32"), residual=s["x"])
    if kind == "topk":
        return s["head"].topk(ops.ln_quantize(s["x"], s["g"], s["b"], 1e-5, "mx32"), case["k"])
    if kind == "mel":
        return ops.power_mel_log(s["spec"], s["mel"], s["mean"], s["istd"])
    if case["mode"] == "graph_ids":
        return s["comp"].run()
    # the eager stack overwrites the features it is given: each pass gets its own copy
    x = s["x"].clone()
    return s["stack"].forward(x, s["pos"]) if case["mode"] == "logits" else s["stack"].forward_ids(x, s["pos"])


def work(case):
    kind = case["kind"]
    if kind in ("dense", "blkscale"):
        m, n, k = case["rows"], case["n"], case["k"]
        bits = BITS["rowscale" if kind == "dense" else "blk16"]
        size = 4 if case.get("dtype") == "float32" else 2
        return {"bytes": m * k * size + n * k * bits / 8 + 4 * n + m * n * 4, "flops": 2 * m * n * k}
    if kind == "mel":
        t, f, m = case["frames"], case["bins"], case["mels"]
        return {"bytes": t * f * 8 + t * m * 4 + m * f * 4, "flops": 2 * t * f * m + 3 * t * f}
    t = case["frames"]
    if kind == "linear":
        n, no = (2 * D, D) if case["op"] == "glu" else (3 * D, 3 * D)
        return {"bytes": t * D * 2 + n * D * BITS[case["fmt"]] / 8 + t * no * 2, "flops": 2 * t * D * n}
    if kind == "ffn":
        return {"bytes": t * D * 4 + 2 * D * FFN * BITS[case["fmt"]] / 8, "flops": 4 * t * D * FFN}
    if kind == "attention":
        return {"bytes": t * D * 6 + 5 * D * D * BITS["mx32"] / 8, "flops": 2 * t * D * 5 * D + 6 * t * t * D}
    if kind == "topk":
        return {"bytes": t * D * 2 + VOCAB * D * BITS["mx32"] / 8 + t * case["k"] * 12, "flops": 2 * t * D * VOCAB}
    weights = (12 * (4 * D * FFN + 8 * D * D) + D * VOCAB) * BITS["mx32"] / 8
    out = t * VOCAB * 2 if case["mode"] == "logits" else t * 4
    return {"bytes": t * D * 4 + weights + out, "flops": t * StackConfig().flops_per_frame()}


def tolerance(case):
    kind = case["kind"]
    if kind in ("dense", "blkscale"):
        return {"rel": 1e-5}  # products of E2M1 codes and powers of two, summed and kept in fp32
    if kind == "topk":
        return {"rel": 1e-5, "differ": 1e-3}  # bf16 logits, log-sum-exp in fp32; equal logits may trade places
    if kind == "mel":
        return {"rel": 1e-3}  # tf32 operands: 2^-10 of the sum under the logarithm
    if kind == "stack" and case["mode"] != "logits":
        return {"differ": 1e-3}  # greedy ids: 99.9 % per-frame agreement
    return {"rel": 1e-2}  # bf16 results
