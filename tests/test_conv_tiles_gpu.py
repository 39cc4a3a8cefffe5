"""The float32 convolution over the edges of its tiles, against float64."""

import pytest
import torch

from citrus_gb300 import _lib

pytestmark = pytest.mark.gpu


def _bound(x, w, bias, k):
    """|error| of a float32 sum of fused multiply-adds: one rounding per product at most, at a partial sum of at most
    the sum of magnitudes."""
    terms = w[0].numel()
    magnitude = torch.nn.functional.conv3d(x.abs(), w.abs(), bias.abs(), padding=k // 2)
    return (terms + 4) * 2.0 ** -24 * magnitude


# voxels around 64 and 128 per tile, channels around 32, fewer channels than the four parts of a split sum, and volumes
# with enough tiles for each of the three forms
@pytest.mark.parametrize("B,shape,ca,cb,co", [
    (1, (2, 2, 2), 1, 0, 1), (2, (2, 4, 4), 3, 0, 31), (1, (4, 4, 4), 2, 3, 33), (3, (2, 6, 4), 5, 2, 12),
    (1, (16, 16, 32), 3, 0, 32), (1, (16, 20, 26), 4, 6, 64), (2, (18, 20, 26), 7, 4, 32)])
@pytest.mark.parametrize("k", [1, 3])
@pytest.mark.parametrize("up", [0, 1])
def test_float32_convolution_and_input_gradient(cuda_device, B, shape, ca, cb, co, k, up):
    gen = torch.Generator(device=cuda_device).manual_seed(ca * 100 + co)
    rand = lambda *s: torch.rand(*s, generator=gen, device=cuda_device) - 0.5  # noqa: E731
    half = [n // 2 for n in shape]
    a, b = rand(B, ca, *shape), rand(B, cb, *(half if up else shape)) if cb else None
    w, bias = rand(co, ca + cb, k, k, k).bfloat16(), rand(co)
    out = torch.empty(B, co, *shape, device=cuda_device)
    error = torch.zeros(1, dtype=torch.int32, device=cuda_device)
    stream = _lib.stream_handle(cuda_device)
    _lib.call("citrus_conv3d_forward_config", a.data_ptr(), ca, _lib.ptr(b), cb, up if cb else 0, w.data_ptr(),
              bias.data_ptr(), out.data_ptr(), co, B, *shape, k, 1, 1, error.data_ptr(), stream)
    x = a.double()
    if cb:
        fine = torch.nn.functional.interpolate(b.double(), scale_factor=2, mode="nearest") if up else b.double()
        x = torch.cat([x, fine], 1)
    wd, bd = w.double(), bias.double()
    ref = torch.relu(torch.nn.functional.conv3d(x, wd, bd, padding=k // 2))
    assert bool(((out.double() - ref).abs() <= _bound(x, wd, bd, k)).all())
    # the input gradient: the transposed convolution of g, split back into the two inputs, the first masked
    g, ga, gb = rand(B, co, *shape), torch.empty_like(a), torch.empty(B, cb, *shape, device=cuda_device) if cb else None
    _lib.call("citrus_conv3d_backward_input_config", g.data_ptr(), co, w.data_ptr(), ga.data_ptr(), ca, a.data_ptr(),
              _lib.ptr(gb), cb, B, *shape, k, 1, error.data_ptr(), stream)
    wt = wd.transpose(0, 1).flip(2, 3, 4)
    grad = torch.nn.functional.conv3d(g.double(), wt, padding=k // 2)
    bound = _bound(g.double(), wt, torch.zeros(ca + cb, device=cuda_device, dtype=torch.float64), k)
    mask = (a > 0).double()
    assert bool(((ga.double() - grad[:, :ca] * mask).abs() <= bound[:, :ca]).all())
    if cb:
        assert bool(((gb.double() - grad[:, ca:]).abs() <= bound[:, ca:]).all())
