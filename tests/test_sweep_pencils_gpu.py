"""The pencil schedule of the sweep gives the per-plane kernel's store bit for bit (the same operations in the same
order, each rounded on its own), so the comparison is exact."""

import numpy as np
import pytest
import torch

from citrus_gb300 import kernels
from citrus_gb300.geometry import Grid
from citrus_gb300.quadrature import product_quadrature
from citrus_gb300.transport_sweep import make_sweep_context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape, G, V, tile, dpb", [
    ((5, 7, 6), 3, 2, 2, 1),         # tiles that do not divide the grid, run-time group count
    ((16, 16, 16), 8, 2, 8, 1),      # whole tiles
    ((9, 17, 11), 8, 3, 8, 1),       # one pencil past a tile, an odd number of views
    ((17, 8, 2), 1, 1, 8, 2),        # fewer slices than loads in flight, directions per task that do not divide
    ((4, 3, 1), 1, 1, 4, 3),         # one slice
    ((1, 1, 37), 5, 1, 4, 3),        # a single pencil
    ((33, 2, 9), 16, 2, 4, 2),       # 512 threads
    ((3, 20, 5), 1, 2, 16, 2),       # the largest tile
    ((6, 6, 6), 170, 1, 1, 1),       # one pencil per block
    ((13, 25, 4), 3, 1, 12, 1),      # a last warp of 16 threads
    ((20, 11, 3), 1, 2, 2, 2),       # 10 x 6 tiles: diagonals that grow, stay and shrink
    ((7, 22, 3), 2, 1, 2, 1),        # 4 x 11 tiles
])
def test_pencil_sweep_equals_per_plane_sweep_bitwise(cuda_device, shape, G, V, tile, dpb):
    rng = np.random.default_rng(sum(shape) + G)
    ctx = make_sweep_context(Grid(shape, 0.5), product_quadrature(4, 12), 2, cuda_device)
    N, D8 = ctx.num_cells, ctx.directions_per_octant
    mu = torch.as_tensor(rng.random((N, G)) + 0.1, dtype=torch.float32, device=cuda_device)
    c = ctx.c.contiguous()
    stores = torch.as_tensor(rng.standard_normal((V, 8, D8, N, 4 * G)), dtype=torch.float32, device=cuda_device)
    expected = stores.clone()
    for v in range(V):
        kernels.sweep_planes(ctx.flat_index, expected[v], mu, c, method="planes")
    for views_per_thread in (1, 2):
        for max_blocks in (0, 1):
            got = stores.clone()
            sync = kernels.sweep_pencils(shape, got, mu, c, tile=tile, dirs_per_block=min(dpb, D8),
                                         views_per_thread=views_per_thread, max_blocks=max_blocks)
            assert torch.equal(got, expected), (views_per_thread, max_blocks)
            assert int(sync[2]) == 0


def test_pencil_wait_that_runs_out_is_reported(cuda_device):
    """A block that never reports its tasks: the next task's wait ends after the limit, the kernel returns with the
    error word set, and the next launch runs normally."""
    ctx = make_sweep_context(Grid((8, 8, 8), 1.0), product_quadrature(2, 4), 1, cuda_device)
    N, G = ctx.num_cells, 2
    store = torch.zeros(8, 1, N, 4 * G, device=cuda_device)
    mu = torch.ones(N, G, device=cuda_device)
    sync = kernels.sweep_pencils(ctx.shape, store, mu, ctx.c.contiguous(), tile=4, max_blocks=1,
                                 timeout_ns=20_000_000, skip_block=0)
    torch.cuda.synchronize()
    assert int(sync[2]) != 0
    ok = kernels.sweep_pencils(ctx.shape, store, mu, ctx.c.contiguous(), tile=4, max_blocks=1)
    torch.cuda.synchronize()
    assert int(ok[2]) == 0


def test_pencil_sweep_rejects_what_it_cannot_take(cuda_device):
    ctx = make_sweep_context(Grid((4, 4, 4), 1.0), product_quadrature(2, 4), 1, cuda_device)
    store = torch.zeros(8, 1, 64, 4 * 8, device=cuda_device)
    mu, c = torch.ones(64, 8, device=cuda_device), ctx.c.contiguous()
    sync = torch.zeros(8, dtype=torch.int32, device=cuda_device)
    for kwargs in (dict(tile=9), dict(dirs_per_block=2), dict(views_per_thread=3), dict(tile=4, sync=sync)):
        with pytest.raises(kernels._lib.CitrusKernelError):
            kernels.sweep_pencils(ctx.shape, store, mu, c, **kwargs)
    with pytest.raises(ValueError):
        kernels.sweep_pencils((4, 4, 5), store, mu, c)


def test_waiting_tasks_outlast_the_limit_while_others_progress(cuda_device):
    """The limit is on the time without progress: the last of the tiles waits for all those before it, here some 20 ms
    with a limit of 5 ms, of which a tile takes a fraction."""
    ctx = make_sweep_context(Grid((1, 64, 4096), 1.0), product_quadrature(2, 4), 1, cuda_device)
    N, G = ctx.num_cells, 1
    gen = torch.Generator().manual_seed(5)
    store = torch.randn(8, 1, N, 4 * G, generator=gen).to(cuda_device)
    mu = (torch.rand(N, G, generator=gen) + 0.1).to(cuda_device)
    expected = store.clone()
    kernels.sweep_planes(ctx.flat_index, expected, mu, ctx.c.contiguous())
    sync = kernels.sweep_pencils(ctx.shape, store, mu, ctx.c.contiguous(), tile=2, timeout_ns=5_000_000)
    assert int(sync[2]) == 0
    assert torch.equal(store, expected)
