"""The oblique projection of several channels at once against each channel count's general form: sums of a channel do not
depend on the others, so a field is projected as part of a wider one (a channel count without a kernel of its own) and
compared exactly."""

import pytest
import torch

from citrus_gb300.geometry import ConeGeometry, Grid
from citrus_gb300.ray_tracing import GB300Projectors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("channels", [2, 3, 4, 5, 6, 7, 8, 12, 16])
@pytest.mark.parametrize("curved", [False, True])
def test_known_channel_counts_equal_the_general_form(cuda_device, channels, curved):
    grid, geo = Grid((7, 9, 11), 0.9), ConeGeometry(60.0, 90.0, 13, 17, 0.9, 0.9, use_curved_detector=curved)
    gen = torch.Generator().manual_seed(channels)
    w = torch.randn(6, 3, generator=gen)
    w = (w / w.norm(dim=1, keepdim=True)).to(cuda_device)
    field = torch.rand(6, 17, *grid.shape, generator=gen).to(cuda_device)  # 17 channels: the general form
    p = GB300Projectors()
    wide = p.oblique_project(field, grid, geo, 0.4, w)
    own = p.oblique_project(field[:, :channels].contiguous(), grid, geo, 0.4, w)
    assert torch.equal(own, wide[:, :channels])
