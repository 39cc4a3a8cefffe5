"""The float32 convolution by bricks, on both sides of the rule that chooses it, against float64."""

import pytest
import torch

import test_conv_tiles_gpu as tiles
from citrus_gb300 import _lib

pytestmark = pytest.mark.gpu


# 3^3: up to 16 output channels and 288 bricks (parts of bricks at every edge), 17 of them; up to 4 input channels and 128 bricks, one
# channel more. 1^3: up to 4 input channels; up to 8 and 16 output channels with 288 bricks, one more of each, and few bricks
@pytest.mark.parametrize("k,B,shape,ca,cb,co,up", [
    (3, 1, (46, 46, 30), 12, 0, 16, 0), (3, 1, (46, 46, 30), 5, 9, 3, 1), (3, 1, (48, 48, 32), 16, 0, 17, 0),
    (3, 2, (14, 32, 32), 4, 0, 8, 0), (3, 1, (27, 35, 31), 3, 0, 16, 0), (3, 2, (13, 27, 31), 5, 0, 7, 0),
    (1, 1, (5, 9, 11), 1, 0, 1, 0), (1, 2, (6, 10, 10), 1, 3, 40, 1), (1, 1, (23, 45, 59), 8, 0, 16, 0),
    (1, 1, (22, 46, 60), 4, 3, 9, 1), (1, 1, (23, 45, 59), 9, 0, 16, 0), (1, 1, (23, 45, 59), 8, 0, 17, 0),
    (1, 1, (5, 9, 11), 8, 0, 16, 0)])
def test_convolution_by_bricks(cuda_device, k, B, shape, ca, cb, co, up):
    tiles.test_float32_convolution_and_input_gradient(cuda_device, B, shape, ca, cb, co, k, up)


def test_more_weights_than_32_bits_index(cuda_device):
    """2^31 weights and more: a 1^3 layer of one voxel, its last output channel read from past the 32-bit offsets."""
    ci, co = 4096, 524289
    w = torch.zeros(co, ci, dtype=torch.bfloat16, device=cuda_device)
    w[0, 0], w[-1, -1], w[-1, 0] = 3.0, 2.0, 0.5
    x = torch.arange(1, ci + 1, dtype=torch.float32, device=cuda_device)
    out = torch.empty(co, device=cuda_device)
    error = torch.zeros(1, dtype=torch.int32, device=cuda_device)
    _lib.call("citrus_conv3d_forward_config", x.data_ptr(), ci, None, 0, 0, w.data_ptr(), None, out.data_ptr(), co, 1, 1, 1,
              1, 1, 0, 1, error.data_ptr(), _lib.stream_handle(cuda_device))
    assert float(out[0]) == 3.0 and float(out[-1]) == 2.0 * ci + 0.5
    assert int((out != 0).sum()) == 2
