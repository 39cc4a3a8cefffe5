"""3^3 weight gradients against float64 autograd. A gradient is a sum of up to 2 x 13 x 9 x 17 products of unit normals in
float32, in a few partial sums: its error is some ten roundings of the largest gradient, 1e-5 of it at most."""

import pytest
import torch
import torch.nn.functional as F

from conftest import rel_err
from citrus_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("co, ca, cb, up", [(1, 1, 0, False), (16, 16, 0, False), (17, 15, 0, False), (33, 3, 14, False),
                                            (16, 8, 25, True)])  # parts of, whole and past a tile of channels
@pytest.mark.parametrize("shape", [(2, 2, 2), (4, 8, 8), (6, 10, 18), (13, 9, 17)])  # parts of, whole and past a brick
@pytest.mark.parametrize("split", [True, False])
def test_weight_gradient_matches_autograd(cuda_device, co, ca, cb, up, shape, split):
    if up and any(n % 2 for n in shape):
        pytest.skip("an upsampled input needs even sizes")
    gen = torch.Generator().manual_seed(co + ca + sum(shape))
    D, H, W = shape
    rand = lambda *s: torch.randn(*s, generator=gen)  # noqa: E731
    a = rand(2, ca, D, H, W)
    b = rand(2, cb, *((n // 2 for n in shape) if up else shape)) if cb else None
    g = rand(2, co, D, H, W)
    x = a if b is None else torch.cat([a, F.interpolate(b, scale_factor=2) if up else b], dim=1)
    w = torch.zeros(co, ca + cb, 3, 3, 3, dtype=torch.float64, requires_grad=True)
    F.conv3d(x.double(), w, padding=1).backward(g.double())
    dev = lambda t: None if t is None else t.to(cuda_device).contiguous()  # noqa: E731
    da, db, dg = dev(a), dev(b), dev(g)
    gw = torch.full((co, ca + cb, 27), float("nan"), device=cuda_device)
    splits = int(_lib.library().citrus_conv3d_weight_grad_splits(co, ca, cb, 2, D, H, W, 3))
    partial = torch.empty(splits * gw.numel(), device=cuda_device) if split else None
    _lib.call("citrus_conv3d_backward_weight", dg.data_ptr(), co, da.data_ptr(), ca, None if db is None else db.data_ptr(),
              cb, int(up), gw.data_ptr(), None, 2, D, H, W, 3, None if partial is None else partial.data_ptr(),
              0 if partial is None else partial.numel(), _lib.stream_handle(cuda_device))
    assert rel_err(gw, w.grad.reshape(co, ca + cb, 27).numpy()) < 1e-5
