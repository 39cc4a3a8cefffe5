"""Inner dimensions above 64 on the tensor cores: two parts in one launch against two launches that accumulate. The parts'
sums are added in the same order, so the comparison is exact."""

import numpy as np
import pytest
import torch

from citrus_gb300 import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M, K, J, batch", [(36, 65, 128, 1),       # one row past a part
                                            (64, 120, 1028, 2),     # a last part of 56 rows, a ragged last tile
                                            (128, 128, 60000, 1),   # whole parts, four accumulators of 128 columns,
                                            (17, 80, 100000, 1),    # and several tiles per block
                                            (100, 129, 516, 1),     # past what one call takes
                                            (70, 96, 333, 1)])      # rows that no bulk copy can read
@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("form", ["ws", "single"])
def test_parts_equal_accumulating_calls(cuda_device, monkeypatch, M, K, J, batch, accumulate, form):
    monkeypatch.setenv("CITRUS_TC_FORM", form)
    rng = np.random.default_rng(M + K)
    dev = lambda *shape: torch.as_tensor(rng.standard_normal(shape), dtype=torch.float32, device=cuda_device)  # noqa: E731
    A, B, C0 = dev(M, K), dev(batch, K, J), dev(batch, M, J)
    err = torch.zeros(1, dtype=torch.int32, device=cuda_device)
    got, want = C0.clone(), C0.clone()
    kernels.small_k_gemm(A, B, got, accumulate=accumulate, precision="bf16x3", error_word=err)
    for k0 in range(0, K, 64):
        kernels.small_k_gemm(A[:, k0:k0 + 64].contiguous(), B[:, k0:k0 + 64], want, accumulate=accumulate or k0 > 0,
                             precision="bf16x3", error_word=err)
    assert int(err[0]) == 0
    assert torch.equal(got, want)
