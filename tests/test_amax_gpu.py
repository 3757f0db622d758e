"""max |x| at the edges of its launch plans (one block or many, eight / four / single loads per turn) and over strided rows."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,cols", [(1, 8), (7, 8), (64, 512), (511, 512), (512, 512), (513, 512), (1025, 264), (4099, 512)])
def test_amax_finds_the_largest_wherever_it_is(dtype, rows, cols):
    from velox_voice_b200 import ops

    x = torch.randn(rows, cols, device="cuda").to(dtype)
    wide = torch.randn(rows, cols + 64, device="cuda").to(dtype) * 100  # what lies between strided rows does not count
    for at in (0, rows * cols // 3, rows * cols - 1):
        y = x.clone()
        y.view(-1)[at] = -77.0
        assert ops.amax(y).item() == 77.0
        wide[:, :cols] = y
        assert ops.amax(wide[:, :cols]).item() == 77.0
    assert ops.amax(torch.zeros_like(x)).item() == 0.0
    y[0, 0] = float("nan")  # a NaN is left out, an infinity is not
    assert ops.amax(y).item() == 77.0
    y[-1, -1] = float("-inf")
    assert ops.amax(y).item() == float("inf")
