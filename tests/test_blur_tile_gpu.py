"""The box blur of adjacent lines (taken in tiles) against the same lines laid out one after another: one warp per line with
the same operations in the same order in both, so the comparison is exact."""

import pytest
import torch

from citrus_gb300 import _lib

pytestmark = pytest.mark.gpu


def _blur(x, strides, lines, length, widths):
    out = torch.full_like(x, float("nan"))
    _lib.call("citrus_box_blur", x.data_ptr(), out.data_ptr(), x.shape[0], lines, length, *strides, *strides,
              widths.data_ptr(), None, None, 1, 0.0, 0.0, _lib.stream_handle(x.device))
    return out


@pytest.mark.parametrize("lines", [1, 15, 16, 83])       # a part of a tile, a tile, tiles and a part
@pytest.mark.parametrize("length", [1, 31, 64, 440, 441])  # 441: past the tiles
def test_adjacent_lines_equal_separate_lines(cuda_device, lines, length):
    gen = torch.Generator().manual_seed(lines + length)
    x = torch.rand(5, length, lines, generator=gen).to(cuda_device)
    widths = torch.tensor([0.0, 0.7, 3.2, 12.5, 2000.0], device=cuda_device)
    tiled = _blur(x, (length * lines, 1, lines), lines, length, widths)
    apart = _blur(x.transpose(1, 2).contiguous(), (length * lines, length, 1), lines, length, widths)
    assert torch.equal(tiled, apart.transpose(1, 2))
