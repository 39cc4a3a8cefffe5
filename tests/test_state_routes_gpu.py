"""The accumulator's encoding on both sides of its rules: one launch for small or cell-adjacent accumulators, tiles else."""

import pytest
import torch

from citrus_gb300 import _lib
from citrus_gb300.state_store import StateStore

pytestmark = pytest.mark.gpu


# adjacent cells (or one group): fewer than 20 (group, moment)s take one launch up to 49152 cells; adjacent groups up to
# 65536 values per moment and 25 MB; two groups with 64 (group, moment)s always
@pytest.mark.parametrize("groups,moments,cells,cell_major,launches", [
    (1, 4, (12, 12, 12), True, 1), (1, 4, (3, 128, 128), True, 1), (1, 4, (1, 193, 255), True, 3),
    (1, 4, (1, 193, 255), False, 3), (5, 4, (1, 193, 255), False, 1), (3, 4, (16, 64, 49), False, 3),
    (8, 4, (16, 16, 16), True, 1), (8, 16, (16, 16, 32), True, 1), (8, 4, (1, 83, 101), True, 3),
    (33, 4, (1, 5, 401), True, 3), (16, 4, (1, 1, 4097), True, 3), (2, 32, (1, 200, 200), True, 1),
    (2, 31, (1, 200, 200), True, 3)])
def test_encoding_takes_one_launch_where_that_is_faster(cuda_device, groups, moments, cells, cell_major, launches):
    """The launches of one encoding, and its codes and scales bit for bit those of the float32 tensor arithmetic."""
    gen = torch.Generator(device=cuda_device).manual_seed(groups)
    phi = 1e-6 * torch.randn(moments, *cells, groups, 4, generator=gen, device=cuda_device)
    phi[1, 0, 0, 0, 0, 0] = float("nan")
    phi[2, -1, -1, -1, -1, 0] = -float("inf")
    phi[3, ..., 0] = -0.0
    phi = phi.permute(4, 0, 5, 1, 2, 3)
    if not cell_major:
        phi = phi.contiguous()
    store = StateStore(1, phi.shape, cuda_device, location="gpu")
    before = _lib.launch_count()
    store.put(0, phi)
    assert _lib.launch_count() - before == launches
    mean = phi[:, :, :1]
    maximum = mean.abs().amax(dim=(2, 3, 4, 5), keepdim=True)
    scale = torch.where(maximum > 0, maximum / 2.0 ** 14, torch.ones_like(maximum))
    stored = (mean / scale).to(torch.float16)
    assert torch.equal(store._scale[0].view(torch.int32), scale.view(torch.int32))
    assert torch.equal(store._data[0].float().nan_to_num(nan=1e5), stored.float().nan_to_num(nan=1e5))
    out = store.get(0)
    assert torch.equal(out[:, :, :1].nan_to_num(nan=1e5), (stored.float() * scale).nan_to_num(nan=1e5))
    assert not bool(out[:, :, 1:].any())
