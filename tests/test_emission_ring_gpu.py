"""The image's emission with its nodes in a ring: blocks that fit it, blocks that do not, and several rounds of it."""

import numpy as np
import pytest
import torch

from test_emission_kernels_gpu import _emission

pytestmark = pytest.mark.gpu


# directions around the 256 of a block; 1, 2, 4, 8 and 16 padded groups (512, 256, 128 and 64 nodes in the ring); the
# points of a block 11 cm apart, which 401 nodes (of 0.005) spread over about 26 nodes
@pytest.mark.parametrize("groups, q, traced, signal, K", [
    (1, 1, True, True, 255), (2, 2, False, True, 256), (4, 1, True, False, 257), (5, 2, True, True, 300),
    (3, 1, True, False, 260), (6, 1, True, True, 260), (7, 2, True, True, 260), (12, 1, True, False, 260),
    (8, 1, True, True, 513), (16, 1, True, True, 260), (16, 2, False, False, 30)])
@pytest.mark.parametrize("num_eta", [2, 101, 401, 2001])
def test_ring_equals_group_lanes(cuda_device, monkeypatch, groups, q, traced, signal, K, num_eta):
    """Bit for bit the group-lane kernel, which reads the table's rows per direction: at 2 nodes one window holds the
    table, at 2001 the points of a block lie too far apart for the ring."""
    import test_emission_kernels_gpu as base
    library = base.spectral_library
    monkeypatch.setattr(base, "spectral_library", lambda *a, **kw: library(*a, **dict(kw, num_eta=num_eta)))
    monkeypatch.delenv("CITRUS_EMISSION_KERNEL", raising=False)
    new = _emission(cuda_device, groups, q, traced, signal, K)
    monkeypatch.setenv("CITRUS_EMISSION_KERNEL", "groups")
    old = _emission(cuda_device, groups, q, traced, signal, K)
    for a, b in zip(new, old):
        assert torch.equal(a, b)
    assert np.isfinite(float(new[0].sum()))
