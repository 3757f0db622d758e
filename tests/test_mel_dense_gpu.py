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
