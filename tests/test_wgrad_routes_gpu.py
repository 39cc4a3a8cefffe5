"""3^3 weight gradients past the rule for one thread per tap, and the workspace of their partial sums."""

import pytest
import torch

import test_wgrad_tiles_gpu as tiles
from citrus_gb300 import _lib

pytestmark = pytest.mark.gpu


# more than 304 blocks of 8 input channels and one brick: parts of, whole and past a tile of 16 channels and of a brick
@pytest.mark.parametrize("co, ca, cb, up, shape", [
    (17, 15, 0, False, (13, 17, 33)), (33, 3, 14, False, (13, 9, 41)), (16, 8, 25, True, (14, 18, 34)),
    (16, 16, 0, False, (20, 40, 33)), (12, 9, 0, False, (26, 33, 33)), (16, 8, 0, False, (26, 33, 33))])
@pytest.mark.parametrize("split", [True, False])
def test_weight_gradient_of_many_bricks(cuda_device, co, ca, cb, up, shape, split):
    tiles.test_weight_gradient_matches_autograd(cuda_device, co, ca, cb, up, shape, split)


@pytest.mark.parametrize("co, ca, cb, batch, shape", [
    (64, 64, 0, 4, (48, 48, 32)), (128, 128, 256, 4, (24, 24, 16)), (128, 128, 0, 1, (48, 48, 32)),
    (32, 32, 64, 4, (24, 24, 16)), (256, 256, 0, 4, (12, 12, 8))])
def test_partial_sums_stay_small(cuda_device, co, ca, cb, batch, shape):
    """At most 64 MB of partial sums."""
    splits = int(_lib.library().citrus_conv3d_weight_grad_splits(co, ca, cb, batch, *shape, 3))
    assert splits > 1 and 4 * splits * co * (ca + cb) * 27 <= 64e6
