"""The small-K products with four columns per thread give the bits of those with two."""

import pytest
import torch

from citrus_gb300 import _lib, kernels

pytestmark = pytest.mark.gpu


# inner dimensions and rows around the unrolled 16, 32 and 36 and the 128 rows of a block; columns past the rule's
# least number that leave one quad in the last block
@pytest.mark.parametrize("M,K", [(1, 1), (5, 16), (128, 17), (131, 32), (120, 36), (16, 120), (17, 65), (33, 120), (36, 121)])
@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("batch", [1, 2])
def test_quads_equal_pairs(cuda_device, M, K, accumulate, batch):
    J = 4 * 128 * 2 * torch.cuda.get_device_properties(0).multi_processor_count + 4
    gen = torch.Generator(device=cuda_device).manual_seed(M * 1000 + K)
    rand = lambda *s: torch.rand(*s, generator=gen, device=cuda_device) - 0.5  # noqa: E731
    A, B, C = rand(M, K), rand(batch, K, J + 4), rand(batch, M, J + 4)
    stream = _lib.stream_handle(cuda_device)

    def product(out, offset, columns):
        _lib.call("citrus_small_k_gemm_config", A.data_ptr(), K, B.data_ptr() + 4 * offset, J + 4,
                  out.data_ptr() + 4 * offset, J + 4, M, K, columns, batch, K * (J + 4), M * (J + 4), int(accumulate), 1,
                  0, stream)

    quads, pairs = C.clone(), C.clone()
    product(quads, 0, J)
    product(pairs, 2, J - 4)                      # 8-byte aligned: two columns per thread
    assert torch.equal(quads[..., 2:J - 2], pairs[..., 2:J - 2])
    assert torch.equal(quads[..., J:], C[..., J:])
    ref = A.double() @ B.double()[..., :J] + (C.double()[..., :J] if accumulate else 0.0)
    size = A.double().abs() @ B.double().abs()[..., :J] + C.double().abs()[..., :J]
    assert bool(((quads.double()[..., :J] - ref).abs() <= (K + 2) * 2.0 ** -24 * size).all())


@pytest.mark.parametrize("M,K", [(1, 16), (130, 36), (7, 20)])
def test_quads_with_means_equal_pairs(cuda_device, M, K):
    J = 4 * 128 * 2 * torch.cuda.get_device_properties(0).multi_processor_count + 4
    gen = torch.Generator(device=cuda_device).manual_seed(M + K)
    A, B = torch.rand(M, K, generator=gen, device=cuda_device), torch.rand(1, K, J, generator=gen, device=cuda_device)
    F = torch.rand(1, M, J // 4, generator=gen, device=cuda_device)
    C = kernels.source_expansion_first(A, B, torch.empty(1, M, J, device=cuda_device), F)
    shifted = torch.empty(1, K, J + 2, device=cuda_device)[..., :J]          # rows of a stride that is no multiple of 4
    shifted.copy_(B)
    out = torch.empty(1, M, J + 2, device=cuda_device)
    _lib.call("citrus_source_expansion_first", A.data_ptr(), K, shifted.data_ptr(), J + 2, out.data_ptr(), J + 2,
              F.data_ptr(), J // 4, M, K, J, 1, K * (J + 2), M * (J + 2), M * (J // 4), _lib.stream_handle(cuda_device))
    assert torch.equal(C, out[..., :J])
