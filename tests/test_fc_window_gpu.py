"""The sampling correction's kept source values where a block's points see the source under wide angles and the window of table rows
moves, starts again, or fits one direction per warp only: bit for bit those of the group-lane kernel."""

import numpy as np
import pytest
import torch

from citrus_gb300.cross_sections import BONE, WATER, spectral_library
from citrus_gb300.geometry import ConeGeometry, Grid
from citrus_gb300.quadrature import product_quadrature
from citrus_gb300.uncollided import first_collision_sampling_correction
from citrus_gb300.workloads import bremsstrahlung_spectrum

pytestmark = pytest.mark.gpu


# groups with and without windows and with the counts known or not; a source at 100, 60, 30 and 12 cm of a box 25.6 cm long
@pytest.mark.parametrize("groups, materials", [(1, 2), (3, 3), (4, 1), (4, 2), (4, 7), (5, 2), (5, 4), (6, 3), (7, 2), (8, 1),
                                               (8, 2), (8, 3), (9, 1), (12, 2), (16, 2), (16, 3), (20, 2)])
@pytest.mark.parametrize("distance", [100.0, 60.0, 30.0, 12.0])
@pytest.mark.parametrize("num_eta", [2, 401, 1201])
def test_windows_of_wide_fans(cuda_device, monkeypatch, groups, materials, distance, num_eta):
    _compare(cuda_device, monkeypatch, groups, materials, distance, num_eta, 117)     # a last batch that is not full


# up to 33 directions of 401 nodes take no window below 9 groups; whole batches gather up to 100
@pytest.mark.parametrize("groups, materials", [(4, 3), (5, 2), (6, 3), (7, 2), (8, 1), (8, 2), (11, 2)])
@pytest.mark.parametrize("directions", [1, 7, 33, 34, 100, 101])
def test_few_directions(cuda_device, monkeypatch, groups, materials, directions):
    _compare(cuda_device, monkeypatch, groups, materials, 60.0, 401, directions)


def _compare(cuda_device, monkeypatch, groups, materials, distance, num_eta, directions):
    rng = np.random.default_rng(groups)
    library = spectral_library(np.linspace(120.0, 30.0, groups + 1), bremsstrahlung_spectrum(seed=0),
                               ([WATER, BONE] * 4)[:materials], 1, num_eta=num_eta, fine_per_group=2)
    grid = Grid((3, 3, 32), 0.8)
    dev = lambda x: torch.as_tensor(x, dtype=torch.float32, device=cuda_device)  # noqa: E731
    rho = dev(rng.random((materials, *grid.shape)) * (rng.random((materials, *grid.shape)) < 0.7))
    phi = dev(rng.random((groups, *grid.shape)) + 0.1)
    q = product_quadrature(6, 20)
    omega, weight = dev(q.omega[:directions]), dev(q.weight[:directions])
    geo = ConeGeometry(distance, distance + 50.0, 64, 64, 0.4, 0.4)

    def run():
        return first_collision_sampling_correction(library, rho, phi, grid, geo, 0.9, omega, weight, keep_sums=True,
                                                   keep_cache=True)

    monkeypatch.delenv("CITRUS_FC_KERNEL", raising=False)
    new = run()
    monkeypatch.setenv("CITRUS_FC_KERNEL", "groups")
    old = run()
    assert torch.equal(new.cache, old.cache)
    # up to 117 positive terms in another order, each rounded at a partial sum of at most the whole
    magnitude = (weight.double()[:, None, None] * old.cache.double()).sum(0).view(groups, *grid.shape)
    for i in range(3):
        error = (new.sums[i].double() - old.sums[i].double()).abs()
        assert bool((error <= 2 * 120 * 2.0 ** -24 * magnitude).all())
