"""Sums over directions around their blocks of 64 and their pixels per block."""

import pytest
import torch

from citrus_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [1, 64, 65, 512, 577])
@pytest.mark.parametrize("rows,cols", [(1, 1), (8, 8), (5, 13)])
@pytest.mark.parametrize("accumulate", [0, 1])
def test_direction_sums_equal_one_call_per_block(cuda_device, K, rows, cols, accumulate):
    """Bit for bit the sums of one call per 64 directions, each added to the accumulator in order."""
    gen = torch.Generator(device=cuda_device).manual_seed(K)
    G, stream = 3, _lib.stream_handle(cuda_device)
    image = torch.rand(K, rows, G, cols, generator=gen, device=cuda_device)   # rows outermost, read through strides
    weights = torch.rand(K, G, 1, cols, generator=gen, device=cuda_device)
    start = torch.rand(G, rows, cols, generator=gen, device=cuda_device)
    strides = (rows * G * cols, cols, G * cols, 1)

    def weighted(acc, s, e, add):
        w, img = weights[s:e].contiguous(), image[s:e].contiguous()
        _lib.call("citrus_weighted_direction_sum", img.data_ptr(), e - s, G, rows, cols, *strides, w.data_ptr(), 1, cols,
                  acc.data_ptr(), add, stream)
        torch.cuda.synchronize()

    def plain(acc, s, e, add):
        img = image[s:e].contiguous()
        _lib.call("citrus_sum_directions", img.data_ptr(), e - s, G * rows * cols, G * rows * cols, acc.data_ptr(), add,
                  stream)
        torch.cuda.synchronize()

    for call in (weighted, plain):
        whole, parts = start.clone(), start.clone()
        call(whole, 0, K, accumulate)
        for s in range(0, K, 64):
            call(parts, s, min(K, s + 64), accumulate or int(s > 0))
        assert torch.equal(whole, parts)
        dims = (weights.double() * image.double().permute(0, 2, 1, 3)).sum(0) if call is weighted else \
            image.double().sum(0).view(G, rows, cols)
        ref = dims + (start.double() if accumulate else 0.0)
        # positive terms: blocks of at most 64 rounded sums and one addition per block
        assert bool(((whole.double() - ref).abs() <= (64 + K // 64 + 2) * 2.0 ** -24 * ref).all())
