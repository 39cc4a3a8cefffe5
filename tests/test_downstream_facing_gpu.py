"""Directions that do not face the panel are told on the device as tensor arithmetic tells them."""

import math

import pytest
import torch

from citrus_gb300 import _lib
from citrus_gb300.geometry import ConeGeometry, Grid
from citrus_gb300.ray_tracing import GB300Projectors, HostArgs, _grid_args, _voxel_major, panel_args

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("curved", [False, True])
@pytest.mark.parametrize("channels,voxel_major", [(1, False), (2, True), (3, True), (8, False)])
@pytest.mark.parametrize("walk", ["kept tables", "lattice", "own walk"])
def test_facing_equals_tensor_arithmetic(cuda_device, curved, channels, voxel_major, walk):
    angle = 0.9
    grid, geo = Grid((3, 5, 11), 1.1), ConeGeometry(50.0, 80.0, 8, 8, 1.0, 1.0, use_curved_detector=curved)
    gen = torch.Generator().manual_seed(channels)
    n = torch.tensor(geo.panel_axes(angle)[2], dtype=torch.float64)
    w = torch.randn(200, 3, generator=gen, dtype=torch.float64)
    w[:100] -= (w[:100] @ n)[:, None] * n                    # along the panel to rounding: either sign, or zero
    w[0] = torch.tensor([0.0, 0.0, 1.0])
    w = (w / w.norm(dim=1, keepdim=True)).float().to(cuda_device)
    vol = torch.rand(channels, *grid.shape, device=cuda_device)
    p = GB300Projectors()
    tables = p.crossing_tables(grid, w)
    out = p.downstream_cumulative(vol, grid, geo, angle, w, lattice=walk != "own walk", voxel_major=voxel_major,
                                  crossings=tables if walk == "kept tables" else None)
    nf = [float(v) for v in geo.panel_axes(angle)[2]]
    toward = ((w[:, 0] * -nf[0] + w[:, 1] * -nf[1] + w[:, 2] * -nf[2]) > 0).to(torch.uint8)
    assert 0 < int(toward[:100].sum()) < 100
    host = HostArgs()
    box, dims = _grid_args(host, grid)
    scratch = torch.empty_like(tables)
    V, ref = grid.num_voxels, torch.empty_like(out)
    strides = (V * channels, 1, channels) if voxel_major else (channels * V, V, 1)
    flat = _voxel_major(vol, grid)
    diagonal = math.sqrt(sum(e * e for e in grid.extent)) * (1 + 1e-9) + 1e-9
    _lib.call("citrus_downstream_cumulative", flat.data_ptr(), channels, box, dims, w.data_ptr(), toward.data_ptr(), 200,
              panel_args(host, geo, angle), diagonal, ref.data_ptr(), *strides,
              None if walk == "own walk" else scratch.data_ptr(), 0 if walk == "own walk" else tables.numel(),
              _lib.stream_handle(cuda_device))
    assert torch.equal(out, ref)
