"""The primary's device pass against the host evaluation of the same geometry, source and responses."""

import numpy as np
import pytest
import torch

from citrus_gb300 import scatter_image
from citrus_gb300.cross_sections import synthetic_library
from citrus_gb300.geometry import ConeGeometry
from citrus_gb300.responses import DetectorResponse, FilterMaterial, SourceModel, ideal_counting_response, no_grid

pytestmark = pytest.mark.gpu


def _detector(kind):
    if kind == "counting":
        return ideal_counting_response()
    theta = np.linspace(0.02, 0.3, 5)                    # narrower than the panel's incidences: clamped at both ends
    return DetectorResponse(np.array([20.0, 60.0, 150.0]), theta,
                            np.array([1.0, 2.0, 3.5])[:, None] * (1.0 + np.cos(7 * theta))[None])


# panels around the 128 pixels of a block; one ray, the four of a pass, and nine (three passes, the last of one ray)
@pytest.mark.parametrize("rows,cols,n", [(1, 1, 1), (8, 16, 1), (3, 43, 2), (5, 31, 3)])
@pytest.mark.parametrize("curved", [False, True])
@pytest.mark.parametrize("detector", ["counting", "angles"])
@pytest.mark.parametrize("source", ["plain", "profile", "filter rows", "filter"])
def test_device_primary_equals_the_host_evaluation(cuda_device, monkeypatch, rows, cols, n, curved, detector, source):
    rng = np.random.default_rng(rows * cols + n)
    library = synthetic_library(num_groups=3, legendre_order=1, num_eta=11)
    geo = ConeGeometry(50.0, 80.0, rows, cols, 1.3, 1.1, det_row_offset=0.7, det_channel_offset=-2.0,
                       use_curved_detector=curved)
    models = {"plain": {}, "profile": {"emission_profile": rng.uniform(0.2, 1.0, (rows, cols))}}
    for name, shape in (("filter rows", (rows, cols)), ("filter", (cols,))):
        models[name] = {"filter_material": FilterMaterial("filter", 2.7, lambda e: 5.0 / np.asarray(e)),
                        "filter_thickness_cm": rng.uniform(0.1, 0.5, shape)}
    path = torch.rand(library.num_materials, rows * n, cols * n, device=cuda_device) * 20.0
    args = (library, path, None, geo, 0.7, SourceModel(**models[source]), _detector(detector), no_grid())
    assert scatter_image._primary_on_device(*args[3:4], *args[5:], library)
    out = scatter_image.primary_from_path_lengths(*args)
    monkeypatch.setattr(scatter_image, "_primary_on_device", lambda *a: False)
    ref = scatter_image.primary_from_path_lengths(*args)
    # sums of E positive float32 terms, the mean and three rounded factors on either side; float64 factors
    bound = 2 * (len(library.fine_energy) + n * n + 8) * 2.0 ** -24
    for key in ("fluence", "planar_fluence", "signal_per_group", "signal"):
        assert out[key].shape == ref[key].shape
        assert bool(((out[key] - ref[key]).abs() <= bound * ref[key].abs()).all()), key


def test_other_classes_and_orders_stay_on_the_host():
    class Panel(ConeGeometry):
        pass

    library = synthetic_library(num_groups=3, legendre_order=1, num_eta=11)
    panel = (80.0, 120.0, 4, 5, 1.0, 1.0)
    args = (SourceModel(), ideal_counting_response(), no_grid())
    assert scatter_image._primary_on_device(ConeGeometry(*panel), *args, library)
    assert not scatter_image._primary_on_device(Panel(*panel), *args, library)
    library.fine_group = library.fine_group[::-1].copy()
    assert not scatter_image._primary_on_device(ConeGeometry(*panel), *args, library)
