"""Two channels at once (two rays per thread) against each channel alone (one ray per thread): the same segments in the
same order with the same roundings, so the comparison is exact."""

import pytest
import torch

from citrus_gb300.geometry import ConeGeometry, Grid
from citrus_gb300.ray_tracing import GB300Projectors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(3, 5, 11), (1, 1, 1), (4, 2, 1), (2, 9, 40), (7, 1, 33)])  # (rows, columns, slices)
@pytest.mark.parametrize("curved", [False, True])
@pytest.mark.parametrize("detector", [40.0, 1.5])  # behind the box, and close enough to cut rays inside it
@pytest.mark.parametrize("voxel_major", [False, True])
def test_two_channels_equal_single_channels(cuda_device, shape, curved, detector, voxel_major):
    grid, geo = Grid(shape, 1.1), ConeGeometry(10.0, 10.0 + detector, 8, 8, 1.0, 1.0, use_curved_detector=curved)
    gen = torch.Generator().manual_seed(sum(shape))
    w = torch.randn(60, 3, generator=gen, dtype=torch.float64)
    w[0], w[1], w[2] = torch.eye(3, dtype=torch.float64)
    w = (w / w.norm(dim=1, keepdim=True)).float().to(cuda_device)
    vol = torch.rand(2, *shape, generator=gen).to(cuda_device)
    p = GB300Projectors()
    both, one, two = (p.downstream_cumulative(x, grid, geo, 0.9, w, lattice=True, voxel_major=False)
                      for x in (vol, vol[:1].contiguous(), vol[1:].contiguous()))
    assert torch.equal(both[:, 0], one[:, 0]) and torch.equal(both[:, 1], two[:, 0])
    if voxel_major:
        major = p.downstream_cumulative(vol, grid, geo, 0.9, w, lattice=True, voxel_major=True)
        assert torch.equal(major.reshape(60, -1, 2), both.reshape(60, 2, -1).transpose(1, 2))
