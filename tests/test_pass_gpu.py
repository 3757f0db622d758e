"""All blocks of a short pass in one launch (``vx_pass.cu``) against the separate launches, bit for bit."""

import pytest
import torch

from test_stack_routes_gpu import build

pytestmark = pytest.mark.gpu


def both(stack, x, pos=None, **kw):
    """(logits, hidden) by the one launch and by separate launches, and the launches of each."""
    from velox_voice_b200 import _lib, ops

    limit, out = stack.one_launch_frames, []
    for frames in (limit, 0):
        stack.one_launch_frames = frames
        ops.reset_launch_count()
        out.append((*stack.forward(x.clone(), pos, return_hidden=True, **kw), ops.launch_count()))
    stack.one_launch_frames = limit
    assert _lib.device_status() == 0
    return out


# row blocks of 128: their edges, one and several clusters, the widest pass of eight-CTA clusters or beyond it, the longest pass
@pytest.mark.parametrize("T", [1, 127, 128, 129, 1000, 1800, 2047, 2500, None])
@pytest.mark.parametrize("ffn", [2048, 1024])
def test_one_launch_has_the_bits_of_the_separate_ones(T, ffn):
    stack = build(blocks=2, ffn=ffn)
    T = stack.one_launch_frames if T is None else T
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, 512, generator=g, device="cuda").bfloat16()
    x[T // 2] = 0.0                      # a row without variance
    x[T // 3] *= 1e4
    (got, h, n1), (want, hidden, n0) = both(stack, x)
    assert torch.equal(got, want) and torch.equal(h, hidden)
    assert n1 == 2 and n0 > 20           # the blocks, the head


@pytest.mark.parametrize("blocks", [1, 16, 17])
def test_number_of_blocks(blocks):
    stack = build(blocks=blocks, vocab=64)
    x = torch.randn(200, 512, device="cuda").bfloat16()
    (got, h, n1), (want, hidden, n0) = both(stack, x)
    assert torch.equal(got, want) and torch.equal(h, hidden) and (n1 == n0) == (blocks == 17)


def same(a, b):
    """Equal bits, a NaN being equal to a NaN."""
    return torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(torch.nan_to_num(a, 0.0), torch.nan_to_num(b, 0.0))


@pytest.mark.parametrize("T", [129, 300, 2100])
def test_rows_that_are_not_finite(T):
    """They have the values of the separate launches and stay to themselves."""
    stack = build(blocks=2)
    x = torch.randn(T, 512, device="cuda").bfloat16()
    clean = stack.forward(x.clone())
    x[5, 7], x[T // 2, 0], x[T - 1, 511], x[17] = float("nan"), float("inf"), float("-inf"), 3e38
    (got, h, _), (want, hidden, _) = both(stack, x)
    assert same(got, want) and same(h, hidden)
    keep = torch.ones(T, dtype=torch.bool, device="cuda")
    keep[[5, T // 2, T - 1, 17]] = False
    assert torch.equal(got[keep], clean[keep])


@pytest.mark.parametrize("T", [1, 300, 2100])
def test_weights_that_may_have_just_been_written(T):
    """Without the scales in natural layout a weight is not known to come from the packing quantizer: its loader waits."""
    stack, other = build(blocks=2), build(blocks=2, seed=1)
    x = torch.randn(T, 512, device="cuda").bfloat16()
    for name, layer in stack.p.items():
        layer.q.scales = None
        layer.q.codes.copy_(other.p[name].q.codes)  # ... and this one was, right before the pass
        layer.q.sf.copy_(other.p[name].q.sf)
    (got, h, n1), (want, hidden, n0) = both(stack, x)
    assert torch.equal(got, want) and torch.equal(h, hidden) and n1 == 2 and n0 > 20


@pytest.mark.parametrize("T", [4300, 9000])
@pytest.mark.parametrize("ffn", [2048, 1024])
def test_more_row_blocks_than_clusters(T, ffn):
    """A cluster takes several row blocks in turn: two rounds, and three of which the last is not full."""
    stack = build(blocks=2, ffn=ffn)
    assert T > stack.one_launch_frames
    stack.one_launch_frames = T
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, 512, generator=g, device="cuda").bfloat16()
    for _ in range(3):
        (got, h, n1), (want, hidden, _) = both(stack, x)
        assert torch.equal(got, want) and torch.equal(h, hidden) and n1 == 2


@pytest.mark.parametrize("offset,pitch,refused", [(8, 528, None), (0, 512, None), (4, 520, "x rows must be 16-byte aligned"),
                                                  (0, 516, "x rows must be 16-byte aligned"), (0, 256, "x rows must be 16-byte aligned"),
                                                  (0, 0, "x rows must be 16-byte aligned")])
def test_rows_of_any_address_and_pitch(offset, pitch, refused):
    """Rows of 16-byte pieces take the one launch; others are refused in the words of the separate launches."""
    from velox_voice_b200 import ops
    from velox_voice_b200._lib import VeloxError

    stack = build(blocks=1)
    x = torch.randn(150, 512, device="cuda").bfloat16()
    limit = stack.one_launch_frames
    for frames in (limit, 0):
        stack.one_launch_frames = frames
        view = torch.zeros(150 * max(pitch, 512) + offset, device="cuda", dtype=torch.bfloat16).as_strided((150, 512), (pitch, 1), offset)
        for source in (False, True):
            call = (lambda: stack.forward(torch.empty_like(x), source=view)) if source else lambda: stack.forward(view)
            if refused:
                with pytest.raises(VeloxError, match=refused):
                    call()
                continue
            view.copy_(x)
            ops.reset_launch_count()
            got = call()
            assert ops.launch_count() == (2 if frames else 14)
            assert torch.equal(got, stack.forward(x.clone()))


def test_a_layer_without_bias_runs_separately():
    from velox_voice_b200 import ops
    from velox_voice_b200._lib import VeloxError

    stack = build(blocks=1)
    x = torch.randn(150, 512, device="cuda").bfloat16()
    want = stack.forward(x.clone())
    odd = torch.zeros(513, device="cuda")[1:]
    odd.copy_(stack.p["b0.lo"].bias)
    stack.p["b0.lo"].bias = odd
    with pytest.raises(VeloxError, match="16-byte aligned"):  # as the separate launches refuse it
        stack.forward(x.clone())
    stack.p["b0.lo"].bias = None
    ops.reset_launch_count()
    assert not torch.equal(stack.forward(x.clone()), want) and ops.launch_count() > 10


def test_passes_on_two_streams():
    stack = build(blocks=3)
    xs = [torch.randn(T, 512, device="cuda").bfloat16() for T in (375, 1300)]
    want = [stack.forward(x.clone()) for x in xs]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in xs]
    got = [[], []]
    for _ in range(20):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                got[i].append(stack.forward(xs[i].clone()))
    torch.cuda.synchronize()
    assert all(torch.equal(o, want[i]) for i in range(2) for o in got[i])


def test_a_bias_that_the_launch_before_wrote():
    """A library GEMM triggers the launch behind it early; the pass reads its biases behind that GEMM's end."""
    from velox_voice_b200 import ops

    stack = build(blocks=1, vocab=64)
    x = torch.randn(100, 512, device="cuda").bfloat16()
    w = ops.quantize(torch.randn(2048, 512, device="cuda"), "mx32")
    bias = stack.p["b0.ffm.w1"].bias = torch.zeros(1, 2048, device="cuda")[0]
    acts = [ops.quantize(torch.randn(1, 512, device="cuda"), "mx32") for _ in range(8)]
    want = []
    for a in acts:
        ops.bsgemm(a, w, out=bias[None])
        torch.cuda.synchronize()
        want.append(stack.forward(x.clone()))
    assert not torch.equal(want[0], want[1])
    for _ in range(10):
        got, xs = [], [x.clone() for _ in acts]
        for a, xx in zip(acts, xs):
            ops.bsgemm(a, w, out=bias[None])
            got.append(stack.forward(xx))
        assert all(torch.equal(g, v) for g, v in zip(got, want))
