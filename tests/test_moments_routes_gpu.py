"""Scattering moments by points and by blocks of points, on both sides of the rule between them."""

import pytest
import torch

from citrus_gb300 import kernels

pytestmark = pytest.mark.gpu


# 1 and 2 groups; 3, 4, 5, 6 and 8 groups just inside and past the bytes up to which points take them (cell-major, then
# moment-major), 7 and 8 groups with too few degrees, and points past the 256 of a block
@pytest.mark.parametrize("groups,L,spatial,cell_major", [
    (1, 0, (1, 1, 1), True), (1, 3, (5, 7, 11), True), (2, 2, (1, 16, 17), False), (2, 5, (8, 8, 4), True),
    (3, 3, (40, 40, 40), True), (3, 3, (1, 255, 257), True), (4, 3, (1, 171, 171), True), (4, 3, (1, 171, 172), True),
    (6, 3, (1, 180, 180), True), (6, 3, (1, 180, 181), True), (5, 2, (9, 10, 107), False), (5, 2, (9, 10, 109), False),
    (4, 1, (1, 165, 165), False), (4, 1, (1, 166, 166), False), (7, 3, (3, 5, 17), True), (7, 2, (3, 5, 17), True),
    (8, 3, (1, 97, 100), True), (8, 3, (1, 98, 100), True), (9, 3, (1, 3, 31), True)])
def test_moments_on_both_sides_of_the_rule(cuda_device, groups, L, spatial, cell_major):
    """Against float64: the fused multiply-adds of the incoming groups, each rounded once."""
    gen = torch.Generator(device=cuda_device).manual_seed(groups + L)
    N = (L + 1) ** 2
    transfer = torch.rand(groups, groups, L + 1, *spatial, generator=gen, device=cuda_device) - 0.3
    phi = (torch.rand(N, *spatial, groups, 4, generator=gen, device=cuda_device) - 0.5).permute(4, 0, 5, 1, 2, 3)
    if not cell_major:
        phi = phi.contiguous()
    for p in (phi, phi[:, :, 0]):
        out = kernels.scattering_moments(transfer, p, "cell_major" if p is phi else "contiguous")
        for n in range(N):
            t, x = transfer[:, :, int(n ** 0.5 + 1e-9)].double(), p[:, n].double()
            equation = "abxyz,akxyz->bkxyz" if p is phi else "abxyz,axyz->bxyz"
            ref, magnitude = torch.einsum(equation, t, x), torch.einsum(equation, t.abs(), x.abs())
            error = (out[:, n].double() - ref).abs()
            assert bool((error <= (groups + 1) * 2.0 ** -24 * magnitude).all()), n
