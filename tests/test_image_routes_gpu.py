"""The row blur by tiles, which takes images of at least 2^19 pixels, and the direction sums of large panels, which one thread per
pixel forms: the small images of the other tests reach neither."""

import pytest
import torch

import test_blur_tile_gpu as blur
import test_direction_sums_gpu as sums

pytestmark = pytest.mark.gpu


# a last tile of 1, 15 and 16 lines; one pixel, the longest line of the tiles and one more
@pytest.mark.parametrize("directions,lines,length", [
    (1, 1 << 19, 1), (2, 8465, 31), (9, 911, 64), (5, 240, 440), (5, 241, 441), (1, 1205, 437)])
def test_tiles_equal_separate_lines(cuda_device, directions, lines, length):
    gen = torch.Generator().manual_seed(lines + length)
    x = torch.rand(directions, length, lines, generator=gen).to(cuda_device)
    widths = torch.linspace(0.0, 60.0, directions).to(cuda_device) + 1.5
    tiled = blur._blur(x, (length * lines, 1, lines), lines, length, widths)
    apart = blur._blur(x.transpose(1, 2).contiguous(), (length * lines, length, 1), lines, length, widths)
    assert torch.equal(tiled, apart.transpose(1, 2))


@pytest.mark.parametrize("K", [64, 65, 97, 130])
@pytest.mark.parametrize("rows,cols", [(96, 114), (95, 114), (209, 210), (208, 210)])  # 3 groups: around 32768 and 131072 pixels
@pytest.mark.parametrize("accumulate", [0, 1])
def test_sums_of_large_panels(cuda_device, K, rows, cols, accumulate):
    sums.test_direction_sums_equal_one_call_per_block(cuda_device, K, rows, cols, accumulate)
