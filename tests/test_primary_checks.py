"""What the primary's device pass refuses, before any launch."""

import numpy as np
import pytest
import torch

from citrus_gb300 import _lib, scatter_image
from citrus_gb300.cross_sections import synthetic_library
from citrus_gb300.geometry import ConeGeometry
from citrus_gb300.responses import FilterMaterial, SourceModel, ideal_counting_response, no_grid


@pytest.mark.parametrize("energies", [-1, 1])
def test_filter_attenuation_of_another_number_of_energies(monkeypatch, energies):
    library = synthetic_library(num_groups=3, legendre_order=1, num_eta=11)
    e = library.fine_energy
    library.fine_energy = e[:-1] if energies < 0 else np.append(e, e[-1])
    launches = []
    monkeypatch.setattr(_lib, "upload", lambda a, device, dtype: torch.as_tensor(np.asarray(a)).to(dtype))
    monkeypatch.setattr(_lib, "call", lambda name, *a: launches.append(name))
    monkeypatch.setattr(_lib, "stream_handle", lambda device: 0)
    geo = ConeGeometry(50.0, 80.0, 3, 5, 1.3, 1.1)
    source = SourceModel(filter_material=FilterMaterial("filter", 2.7, lambda e: 5.0 / np.asarray(e)),
                         filter_thickness_cm=np.full((3, 5), 0.2))
    args = (geo, 0.7, source, ideal_counting_response(), no_grid())
    assert scatter_image._primary_on_device(geo, *args[2:], library)
    with pytest.raises(ValueError, match="filter_attenuation has"):
        scatter_image.primary_from_path_lengths(library, torch.rand(library.num_materials, 3, 5), None, *args)
    assert not launches
