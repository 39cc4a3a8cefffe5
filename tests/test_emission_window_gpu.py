"""The image's emission where a block's points see the source under wide angles: nodes in the ring, rows in the window, and rows in
global memory, with one to eight materials, bit for bit the group-lane kernel."""

import numpy as np
import pytest
import torch

from citrus_gb300 import _lib
from citrus_gb300.cross_sections import BONE, WATER, spectral_library
from citrus_gb300.geometry import ConeGeometry, Grid
from citrus_gb300.ray_tracing import HostArgs
from citrus_gb300.uncollided import _FCArgs
from citrus_gb300.workloads import bremsstrahlung_spectrum

pytestmark = pytest.mark.gpu


def _emission(device, groups, materials, distance, K, length, q=1, signal=True, traced=True):
    """A column of 3 x 2 cells, 32 along the axis (25.6 cm): every block's points span all of it."""
    rng = np.random.default_rng(groups + materials)
    dev = lambda x: torch.as_tensor(np.asarray(x), dtype=torch.float32, device=device)  # noqa: E731
    library = spectral_library(np.linspace(120.0, 30.0, groups + 1), bremsstrahlung_spectrum(seed=0),
                               ([WATER, BONE] * 4)[:materials], 1, num_eta=401, fine_per_group=2)
    grid = Grid((3 * q, 2 * q, 32 * q), 0.8 / q)
    V, NC, G = grid.num_voxels, 192, groups
    rho = rng.random((materials, *grid.shape)) * (rng.random((materials, *grid.shape)) < 0.7)  # zeros among them
    fc = _FCArgs(library, dev(rho), dev(rng.random((G, *grid.shape)) + 0.1), grid,
                 ConeGeometry(distance, distance + 50.0, 32, 48, 0.4, 0.4), 0.7)
    u = rng.standard_normal((K, 3))
    omegas = dev(length * u / np.linalg.norm(u, axis=1, keepdims=True))
    TM = materials
    tau, tau_mu = (dev(rng.random((K, NC, TM)) * 6.0), dev(library.mu_t)) if traced else (dev(rng.random((K, NC, G))), None)
    mu, multiple = dev(rng.random((G, NC)) * 0.3), dev(rng.random((K, NC, G)))
    heights, weight = dev(rng.standard_normal(V) * 5.0), dev(rng.random((K, G))) if signal else None
    host = HostArgs()
    out = torch.full((K, V, 1 if signal else G), float("nan"), device=device)
    partial = torch.empty(K * -(-V // 32) * 2, device=device)
    sums = torch.empty(K, 2, device=device)
    _lib.call("citrus_attenuated_emission", *fc.common(), q, host.doubles(grid.deltas), fc.focal, fc.table.data_ptr(),
              fc.num_eta, fc.eta_lo, fc.eta_hi, omegas.data_ptr(), K, tau.data_ptr(), _lib.ptr(tau_mu),
              TM if traced else 0, mu.data_ptr(), multiple.data_ptr(), heights.data_ptr(), _lib.ptr(weight),
              out.data_ptr(), partial.data_ptr(), partial.numel(), sums.data_ptr(), fc.stream)
    torch.cuda.synchronize()
    return out, partial, sums


@pytest.mark.parametrize("groups, materials, options", [
    (1, 2, {}), (2, 1, {}), (3, 2, {"signal": False}), (4, 7, {}), (5, 2, {}), (5, 7, {"q": 2}), (6, 3, {}), (8, 2, {}),
    (8, 1, {"traced": False}), (8, 2, {"q": 2, "signal": False}), (8, 3, {}), (8, 7, {}), (12, 2, {}), (16, 2, {}),
    (16, 3, {"signal": False})])
@pytest.mark.parametrize("distance", [100.0, 60.0, 45.0, 15.0])
@pytest.mark.parametrize("length", [1.0, 2.5])
def test_wide_fans_equal_group_lanes(cuda_device, monkeypatch, groups, materials, options, distance, length):
    """Directions of another length than 1 reach more nodes (their cosines are held at the ends of the table)."""
    monkeypatch.delenv("CITRUS_EMISSION_KERNEL", raising=False)
    new = _emission(cuda_device, groups, materials, distance, 300, length, **options)
    monkeypatch.setenv("CITRUS_EMISSION_KERNEL", "groups")
    old = _emission(cuda_device, groups, materials, distance, 300, length, **options)
    for a, b in zip(new, old):
        assert torch.equal(a, b)
    assert np.isfinite(float(new[0].sum()))
