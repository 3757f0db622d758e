"""The dense filterbank kernel (``power_mel_log_dense_kernel``: contiguous spectrum, at most 128 mel rows and 448 bins)
at the edges of its tiles and of its range, and the shapes next to them that take the general kernel."""

import numpy as np
import pytest
import torch

from oracle import mel as ML

pytestmark = pytest.mark.gpu


# frames: one row, a cut last chunk (odd rows of an odd number of bins leave 8 bytes), around a chunk (8), a tile (32) and a
# round over the SMs; bins: one step of 8, a stage of 32 and their neighbours, the largest; mel rows: 1, a quadrant, 128
@pytest.mark.parametrize("T,F,M", [(1, 257, 80), (7, 33, 1), (8, 8, 33), (9, 31, 128), (31, 257, 128), (32, 32, 32), (33, 9, 80), (63, 447, 96),
                                   (65, 448, 96), (65, 449, 96), (40, 257, 129), (32 * 148 + 1, 257, 80), (2 * 32 * 148 + 15, 129, 65)])
@pytest.mark.parametrize("offset", [0, 1])
def test_edges_match_the_oracle(T, F, M, offset):
    """offset 1: the spectrum starts 8 bytes behind a 16-byte boundary (the general kernel).  Bound: the tensor core
    adds ceil(F / 8) <= 57 groups of products in fp32, each addition off by at most 2^-23 of a non-negative sum (7e-6
    under the logarithm), the logarithm itself adds 5e-7 + 2^-24 |log|, and istd < 1.5 scales both: below 2e-5."""
    from velox_voice_b200 import ops

    rng = np.random.default_rng(T * 1000 + F + M)
    spec = ((rng.standard_normal((T, F)) + 1j * rng.standard_normal((T, F))) * 3.0).astype(np.complex64)
    bank = ML.mel_filterbank(F, M, seed=M)
    mean, istd = rng.standard_normal(M).astype(np.float32), (rng.random(M) + 0.5).astype(np.float32)
    flat = torch.full((T * F + offset,), complex(float("nan"), float("nan")), dtype=torch.complex64, device="cuda")
    flat[offset:] = torch.from_numpy(spec.reshape(-1)).cuda()
    cu = lambda a: torch.from_numpy(a).cuda()
    out = ops.power_mel_log_tf32(flat[offset:].view(T, F), cu(bank), cu(mean), cu(istd)).cpu().numpy()
    assert np.abs(out - ML.power_mel_log_tf32(spec, bank, mean, istd)).max() < 2e-5


# Where the filterbank passes through shared memory and how many chunks come in ahead of it: all slots of the ring (few mel rows, many bins), some, none (a bank that
# reaches over the operand tiles); banks of odd and even pitch, off a 16-byte boundary, with columns between their rows
@pytest.mark.parametrize("T,F,M", [(100, 447, 1), (32 * 148 * 2 + 5, 447, 2), (100, 447, 96), (47, 445, 90), (100, 257, 80), (24, 257, 128), (100, 255, 3), (100, 256, 80), (40, 3, 1), (40, 1, 2)])
@pytest.mark.parametrize("form", ["dense", "shifted", "strided"])
def test_places_of_the_filterbank(T, F, M, form):
    from velox_voice_b200 import ops

    rng = np.random.default_rng(T + F + M)
    spec = ((rng.standard_normal((T, F)) + 1j * rng.standard_normal((T, F))) * 3.0).astype(np.complex64)
    bank = rng.random((M, F)).astype(np.float32)
    wide = torch.full((M * (F + 3) + 1,), float("nan"), device="cuda")
    cu = {"dense": wide[: M * F].view(M, F), "shifted": wide[1 : M * F + 1].view(M, F), "strided": wide[: M * (F + 3)].view(M, F + 3)[:, :F]}[form]
    cu.copy_(torch.from_numpy(bank))
    zero, one = np.zeros(M, np.float32), np.ones(M, np.float32)
    for _ in range(2):  # the second right behind the first
        out = ops.power_mel_log_tf32(torch.from_numpy(spec).cuda(), cu, torch.from_numpy(zero).cuda(), torch.from_numpy(one).cuda())
    assert np.abs(out.cpu().numpy() - ML.power_mel_log_tf32(spec, bank, zero, one)).max() < 2e-5  # as above
