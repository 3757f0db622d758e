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
@pytest.mark.parametrize("by", [float("-inf"), torch.finfo(torch.bfloat16).min, -1e10])
def test_masked_columns(ops, N, masked, by):
    """A bias of -inf, of the lowest bf16 value or of some large negative one masks tokens.  The selection kernel reads 8 columns per lane and step of 256: masked are the first
    8, everything that lane 0 reads, all but 16 columns, everything from the second step on."""
    torch.manual_seed(N)
    M, K = 9, 512
    a = ops.quantize(torch.randn(M, K, device="cuda"), "mx32", natural=False)
    b = ops.quantize(0.05 * torch.randn(N, K, device="cuda"), "mx32")
    bias = torch.randn(N, device="cuda")
    col = torch.arange(N, device="cuda")
    mask = {"first_piece": col < 8, "lane": (col % 256) < 8, "all_but_16": (col % (N // 16)) != 3, "tail": col >= 256}[masked]
    bias[mask] = by
    _check(ops, a, b, bias, 4)


@pytest.mark.parametrize("masked", ["first_chunk", "second_chunk", "group", "half"])
@pytest.mark.parametrize("by", [float("-inf"), torch.finfo(torch.bfloat16).min, -1e10])
@pytest.mark.parametrize("N", [96, 1000, 5538])
def test_log_sum_exp_of_the_arg_max_head_with_masked_columns(ops, N, masked, by):
    """The epilogue sums 32 columns at a time and two such chunks per partial: masked are either chunk, a whole group of 64, and
    every other chunk of the row."""
    torch.manual_seed(N)
    M, K = 140, 512
    a = ops.quantize(torch.randn(M, K, device="cuda"), "mx32", natural=False)
    b = ops.quantize(0.05 * torch.randn(N, K, device="cuda"), "mx32")
    bias = torch.randn(N, device="cuda")
    col = torch.arange(N, device="cuda")
    bias[{"first_chunk": col < 32, "second_chunk": (col // 32) == 1, "group": col < 64, "half": (col // 32) % 2 == 0}[masked]] = by
    ids, lse, logp = ops.bsgemm_argmax(a, b, bias, return_logp=True)
    z = ops.bsgemm(a, b, epilogue=ops.EPI_BIAS, bias=bias, out_dtype=torch.bfloat16).double()
    assert torch.equal(ids.long(), z.argmax(1))
    want = torch.logsumexp(z, 1)  # (ex2 to 2 ulp, |lse| below 16, as above)
    assert (lse.double() - want).abs().max().item() < 4e-5
    assert (logp.double() - (z.max(1).values - want)).abs().max().item() < 4e-5


@pytest.mark.parametrize("by", [torch.finfo(torch.bfloat16).min, -1e10, -1e9, -1e8])
def test_rows_of_masked_columns_only(ops, by):
    """Every logit is the same large negative value: log_softmax is -log N for each."""
    M, N, K = 5, 520, 512
    a = ops.quantize(torch.randn(M, K, device="cuda"), "mx32", natural=False)
    b = ops.quantize(0.05 * torch.randn(N, K, device="cuda"), "mx32")
    bias = torch.full((N,), by, device="cuda")
    z = ops.bsgemm(a, b, epilogue=ops.EPI_BIAS, bias=bias, out_dtype=torch.bfloat16)
    assert (z == z[0, 0]).all()
    logp, ids = ops.bsgemm_topk(a, b, bias, 4)
    assert torch.equal(ids, torch.arange(4, device="cuda").expand(M, 4))
    first, lse, best = ops.bsgemm_argmax(a, b, bias, return_logp=True)
    assert (first == 0).all() and torch.isfinite(best).all()
    assert (lse.double() - torch.logsumexp(z.double(), 1)).abs().max().item() <= 2.0 ** -23 * abs(float(z[0, 0]))
    # the log-sum-exp is an fp32 number of the logits' magnitude: half a unit in its last place
    assert (logp + torch.log(torch.tensor(float(N)))).abs().max().item() <= max(2.0 ** -24 * abs(float(z[0, 0])), 1e-5)


def test_per_16_format(ops):
    torch.manual_seed(6)
    M, N, K = 130, 5538, 512
    a = ops.quantize(torch.randn(M, K, device="cuda"), "blk16_a")
    b = ops.quantize(0.05 * torch.randn(N, K, device="cuda"), "blk16_b")
    _check(ops, a, b, torch.randn(N, device="cuda"), 5)


@pytest.mark.parametrize("M,k,capacity", [(130, 5, 64), (1, 1, 4), (257, 16, 256), (40, 5, 6)])
def test_entry_points_without_logits(ops, M, k, capacity):
    """vx_bsgemm with lse_partials, vx_ctc_topk_threshold, the candidate pass and vx_ctc_topk_finish: the top-k without a
    logits buffer.  A row whose candidates do not fit its list is reported (ids -1) and counted in `overflow`."""
    from velox_voice_b200 import _lib

    torch.manual_seed(M)
    N, K = 5538, 512
    a = ops.quantize(torch.randn(M, K, device="cuda"), "mx32", natural=False)
    b = ops.quantize(0.05 * torch.randn(N, K, device="cuda"), "mx32")
    bias = torch.randn(N, device="cuda")
    lib = _lib.load()
    st = torch.cuda.current_stream().cuda_stream
    parts = torch.empty(int(lib.vx_ctc_lse_parts(N)), M, 2, device="cuda")
    keys = torch.empty(M, dtype=torch.int64, device="cuda")
    thr, logp = torch.empty(M, device="cuda"), torch.empty(M, k, device="cuda")
    cand = torch.empty(M, capacity, dtype=torch.int64, device="cuda")
    cnt, over = torch.zeros(M, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    ids = torch.empty(M, k, dtype=torch.int32, device="cuda")
    d, keep = ops._gemm_desc(a, b, bias)
    d.epilogue, d.out_dtype, d.out, d.ldo, d.lse_partials = ops.EPI_BIAS_ARGMAX, _lib.DT_F32, keys.data_ptr(), 1, parts.data_ptr()
    _lib.check(lib.vx_bsgemm(C.byref(d), st), "vx_bsgemm")
    _lib.check(lib.vx_ctc_topk_threshold(parts.data_ptr(), N, M, k, thr.data_ptr(), st), "vx_ctc_topk_threshold")
    d.topk_threshold, d.topk_candidates, d.topk_count, d.topk_capacity = thr.data_ptr(), cand.data_ptr(), cnt.data_ptr(), capacity
    _lib.check(lib.vx_bsgemm(C.byref(d), st), "vx_bsgemm")
    _lib.check(lib.vx_ctc_topk_finish(cand.data_ptr(), cnt.data_ptr(), capacity, parts.data_ptr(), N, M, k, ids.data_ptr(),
                                      logp.data_ptr(), over.data_ptr(), st), "vx_ctc_topk_finish")
    z = ops.bsgemm(a, b, epilogue=ops.EPI_BIAS, bias=bias, out_dtype=torch.bfloat16)
    n = (z.float() >= thr[:, None]).sum(1)
    assert torch.equal(n.int(), cnt) and int(over) == int((n > capacity).any())
    full = n > capacity
    assert (ids[full] == -1).all()
    want_logp, want_ids = ops.bsgemm_topk(a, b, bias, k)
    assert torch.equal(ids[~full].long(), want_ids[~full])
    # two summation orders of the fp32 log-sum-exp of one row (see _check)
    assert torch.allclose(logp[~full], want_logp[~full], rtol=0, atol=4e-5)
    del keep


@pytest.mark.parametrize("N", [1024, 1032, 1500, 4096, 6137, 6144, 6152])
@pytest.mark.parametrize("k", [1, 7, 16])
def test_widths_around_the_kernels_ranges(ops, N, k):
    """Rows of more than 1,024 and up to 6,144 columns are held in registers, others read twice; equal logits
    (more than a row's candidate list holds) and rows whose columns are masked but for fewer than k."""
    torch.manual_seed(N + k)
    M, K = 67, 512
    a = ops.quantize(torch.randn(M, K, device="cuda"), "mx32", natural=False)
    b = ops.quantize(0.05 * torch.randn(N, K, device="cuda"), "mx32")
    bias = torch.randn(N, device="cuda")
    _check(ops, a, b, bias, k)
    few = torch.full((N,), float("-inf"), device="cuda")
    few[torch.randperm(N, device="cuda")[: k + 3]] = 0.5
    _check(ops, a, b, few, k)
    zero = ops.quantize(torch.zeros(N, K, device="cuda"), "mx32")
    logp, ids = ops.bsgemm_topk(a, zero, torch.full((N,), 2.0, device="cuda"), k)  # all equal: the lowest columns
    assert torch.equal(ids, torch.arange(k, device="cuda").expand(M, k))
    assert (logp + torch.log(torch.tensor(float(N)))).abs().max().item() < 4e-5
    bias[N // 2] = float("nan")  # no column is a NaN's winner, and every log-probability of the row is one
    logp, ids = ops.bsgemm_topk(a, b, bias, k)
    assert torch.isnan(logp).all() and (ids != N // 2).all()


@pytest.mark.parametrize("equal", [60, 100, 200])
def test_a_nan_is_no_winner_among_many_equal_logits(ops, equal):
    """Fewer equal winners than a row's lists hold, more pieces than listed, more columns than listed: the rescans leave a NaN out as
    the lists do."""
    M, N, k = 5, 5538, 6
    a = ops.quantize(torch.randn(M, 512, device="cuda"), "mx32", natural=False)
    zero = ops.quantize(torch.zeros(N, 512, device="cuda"), "mx32")
    bias = torch.zeros(N, device="cuda")
    top = 11 + 24 * torch.arange(equal, device="cuda")  # a piece of its own each
    bias[top], bias[1000] = 2.0, float("nan")
    logp, ids = ops.bsgemm_topk(a, zero, bias, k)
    assert torch.equal(ids, top[:k].expand(M, k)) and torch.isnan(logp).all()


@pytest.mark.parametrize("N", [1500, 5538])
def test_log_probability_of_two_equal_logits(ops, N):
    """Rows held in registers: log(1/2) for logits c in [16, 32): the log-sum-exp c + log 2 is rounded once (2^-20), exponential and logarithm take up to
    3.6e-7, and the rounding of c log2 e (up to 2^-19 log 2) must not come on top."""
    a = ops.quantize(torch.randn(3, 512, device="cuda"), "mx32", natural=False)
    zero = ops.quantize(torch.zeros(N, 512, device="cuda"), "mx32")
    for c in torch.arange(16, 31, 0.125):
        bias = torch.full((N,), float("-inf"), device="cuda")
        bias[7], bias[N // 2] = c, c
        logp, ids = ops.bsgemm_topk(a, zero, bias, 2)
        assert torch.equal(ids, torch.tensor([7, N // 2], device="cuda").expand(3, 2))
        assert (logp.double() + torch.log(torch.tensor(2.0, dtype=torch.float64))).abs().max().item() < 2.0**-20 + 3.6e-7, c


@pytest.mark.parametrize("N", [1025, 1791, 1792, 1793, 1800, 2047, 2048, 2049, 3839, 3841, 4095, 4097, 5887, 5889, 6143])
def test_ragged_last_pieces_of_rows_in_registers(ops, N):
    """The ragged last 8 columns of a row go to the last slot of lane 0 unless another piece is there: both sides of that line for
    rows of up to 8, 16 and 24 pieces a lane, the winner in and around those columns, and lists of one and two entries a lane."""
    torch.manual_seed(N)
    a = ops.quantize(torch.randn(21, 512, device="cuda"), "mx32", natural=False)
    b = ops.quantize(0.05 * torch.randn(N, 512, device="cuda"), "mx32")
    bias = torch.randn(N, device="cuda")
    for k in (1, 5, 16):
        _check(ops, a, b, bias, k)
    for col in (0, N // 8 * 8 - 1, min(N // 8 * 8, N - 1), N - 1):
        one = bias.clone()
        one[col] = 50.0
        assert (ops.bsgemm_topk(a, b, one, 3)[1][:, 0] == col).all()
        _check(ops, a, b, one, 3)
