"""max |x| at the edges of its launch plans (one block or many, eight / four / up to three loads together) and over strided rows."""

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


@pytest.mark.parametrize("dtype,rows", [(torch.bfloat16, 34000), (torch.bfloat16, 45001), (torch.float32, 20003)])
def test_amax_of_a_tensor_walked_in_strides(dtype, rows):
    """More than 34 MB: every block comes round again, eight vectors a turn, then four and up to three; the largest in each of these parts."""
    from velox_voice_b200 import ops

    x = torch.zeros(rows, 512, dtype=dtype, device="cuda")
    threads = torch.cuda.get_device_properties(0).multi_processor_count * 8 * 256
    per = 16 // x.element_size()
    for turn in range(-(-x.numel() // per // threads)):
        at = min((turn * threads + 12345) * per + 3, x.numel() - 1)
        x.view(-1)[at] = -3.0
        assert ops.amax(x).item() == 3.0, turn
        x.view(-1)[at] = 0.0
    x[-1, -1] = 5.0
    assert ops.amax(x).item() == 5.0


@pytest.mark.parametrize("rows", [2368, 2369, 5000])  # up to one block per SM (an atomic maximum per warp), beyond (per block)
def test_amax_either_side_of_one_block_per_sm(rows):
    from velox_voice_b200 import ops

    for dtype in (torch.bfloat16, torch.float32):
        x = torch.randn(rows, 512, device="cuda").to(dtype)
        want = x.float().abs().max()
        assert ops.amax(x) == want
        wide = torch.cat([x, x * 100], dim=1)
        assert ops.amax(wide[:, :512]) == want
