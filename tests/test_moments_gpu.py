"""Scattering moments over the edges of their tiles against a float64 sum."""

import pytest
import torch

from citrus_gb300 import kernels

pytestmark = pytest.mark.gpu


# groups around the unrolled counts (4, 8, 12, 16, 32) and past the 32 outgoing groups of a block; points around 32
@pytest.mark.parametrize("groups_in,groups_out,spatial", [
    (1, 1, (1, 1, 1)), (3, 3, (3, 11, 1)), (4, 4, (2, 4, 4)), (5, 7, (1, 1, 31)), (8, 8, (4, 4, 4)), (9, 9, (1, 5, 13)),
    (13, 16, (1, 3, 11)), (16, 16, (2, 3, 17)), (17, 17, (1, 2, 17)), (32, 37, (1, 1, 33))])
@pytest.mark.parametrize("layout", kernels.LAYOUTS)
@pytest.mark.parametrize("cell_major_in", [True, False])
@pytest.mark.parametrize("linear", [True, False])
def test_scattering_moments_match_float64(cuda_device, groups_in, groups_out, spatial, layout, cell_major_in, linear):
    gen = torch.Generator(device=cuda_device).manual_seed(groups_in * 100 + groups_out)
    L, N = 3, 9                                           # a library of one order more than the moments use
    transfer = torch.rand(groups_in, groups_out, L + 1, *spatial, generator=gen, device=cuda_device) - 0.3
    phi = torch.rand(N, *spatial, groups_in, 4, generator=gen, device=cuda_device) - 0.5
    phi = phi.permute(4, 0, 5, 1, 2, 3) if linear else phi[..., 0].permute(4, 0, 1, 2, 3)
    if not cell_major_in:
        phi = phi.contiguous()
    out = kernels.scattering_moments(transfer, phi, layout)
    degree = torch.tensor([0, 1, 1, 1, 2, 2, 2, 2, 2], device=cuda_device)
    t = transfer.double()[:, :, degree]                   # [G_in, G_out, N, ...]
    equation = "abnxyz,ankxyz->bnkxyz" if linear else "abnxyz,anxyz->bnxyz"
    ref = torch.einsum(equation, t, phi.double())
    magnitude = torch.einsum(equation, t.abs(), phi.double().abs())
    # groups_in fused multiply-adds in float32, each rounded once at a partial sum of at most the magnitude
    assert bool(((out.double() - ref).abs() <= (groups_in + 1) * 2.0 ** -24 * magnitude).all())
