"""Corrected first-collision moments from the kept source values against the same call evaluating the source again: the
same terms of each point in the same order, each within a few float32 roundings, so 1e-6 of the largest moment."""

import numpy as np
import pytest
import torch

from conftest import rel_err
from citrus_gb300.cross_sections import BONE, WATER, spectral_library
from citrus_gb300.geometry import ConeGeometry, Grid
from citrus_gb300.quadrature import product_quadrature
from citrus_gb300.uncollided import first_collision_moments_at_directions, first_collision_sampling_correction
from citrus_gb300.workloads import bremsstrahlung_spectrum

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("groups", [1, 8, 20])  # 20: the points' factors of two per axis are not kept in registers
@pytest.mark.parametrize("factor", [1, 2, 3])
@pytest.mark.parametrize("count", [1, 8, 19])  # directions: a part of, one, and past two unrolled passes
def test_cached_moments_equal_direct_moments(cuda_device, groups, factor, count):
    library = spectral_library(np.linspace(120.0, 30.0, groups + 1), bremsstrahlung_spectrum(seed=0), [WATER, BONE],
                               1, num_eta=201, fine_per_group=2)
    grid = Grid((6, 6, 12), 0.6)  # up to 432 cells: a last block of 16
    geo = ConeGeometry(100.0, 150.0, 64, 64, 0.4, 0.4)
    rng = np.random.default_rng(groups)
    dev = lambda x: torch.as_tensor(x, dtype=torch.float32, device=cuda_device)  # noqa: E731
    rho = dev(rng.random((2, *grid.shape)))
    phi = dev(rng.random((groups, *grid.shape)) * 1e-3 + 1e-4)
    q = product_quadrature(6, 20)
    corr = first_collision_sampling_correction(library, rho, phi, grid, geo, 0.9, dev(q.omega), dev(q.weight),
                                               keep_cache=True)
    rows = torch.as_tensor(rng.permutation(120)[:count], device=cuda_device)
    args = (library, rho, phi, grid, geo, 0.9, dev(q.omega)[rows], corr, factor)
    cached = first_collision_moments_at_directions(*args, cell_major=True, direction_index=rows)
    direct = first_collision_moments_at_directions(*args, cell_major=True)
    assert rel_err(cached, direct) < 1e-6
