"""Memory of the image chunks: a budget that looks at what the device has free, fixed per solver, and counted by the batched sweep."""

from types import SimpleNamespace

import pytest
import torch

from citrus_gb300 import batched, scatter_solver
from citrus_gb300.geometry import ConeGeometry, Grid
from citrus_gb300.scatter_solver import ScatterSolver

GIB = 2 ** 30


@pytest.fixture
def memory(monkeypatch):
    """A device whose memory the test sets."""
    state = SimpleNamespace(free=280 * GIB, cached=0, capturing=False)
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda device=None: (state.free, 284 * GIB))
    monkeypatch.setattr(torch.cuda, "memory_reserved", lambda device=None: state.cached + GIB)
    monkeypatch.setattr(torch.cuda, "memory_allocated", lambda device=None: GIB)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: state.capturing)
    return state


def _solver():
    solver = ScatterSolver.__new__(ScatterSolver)
    solver.library = SimpleNamespace(num_groups=8)
    solver.config = SimpleNamespace(cone_num_polar=16, cone_num_azimuthal=32, direction_chunk=8)
    solver.geometry = ConeGeometry(100.0, 150.0, 192, 256, 0.16, 0.16)
    solver.device = torch.device("cuda")
    solver._image_budget = None
    grid = Grid((64, 64, 64), 0.4)
    return solver, SimpleNamespace(grid_quadrature=grid, grid_coarse=grid)


@pytest.mark.parametrize("free, cached", [(280, 0), (33, 0), (1, 32), (16, 0), (2, 6), (1, 0), (0, 0)])
def test_chunks_fit_a_share_of_the_free_memory(memory, free, cached):
    memory.free, memory.cached = free * GIB, cached * GIB
    solver, fields = _solver()
    chunk = solver.image_direction_chunk(fields)
    used = chunk * solver.image_bytes_per_direction(fields)
    if free + cached >= 32:
        assert chunk == 256                       # of 512: two chunks in 8 GiB
    else:
        assert chunk == 8 or used <= (free + cached) * GIB / 4
    memory.free = 280 * GIB                       # the chunks of a solver stay the same
    assert solver.image_direction_chunk(fields) == chunk


def test_capture_decides_nothing(memory):
    solver, fields = _solver()
    memory.free, memory.capturing = 4 * GIB, True
    assert solver.image_direction_chunk(fields) == 256
    memory.capturing = False
    assert solver.image_direction_chunk(fields) < 256


def test_views_leave_room_for_the_images(memory):
    ctx = SimpleNamespace(num_cells=64 ** 3, num_moments=36)
    memory.free = 100 * GIB
    alone = batched.views_that_fit(ctx, 8, 15, "cuda")
    memory.free = 108 * GIB
    assert batched.views_that_fit(ctx, 8, 15, "cuda", image_bytes=8 * GIB) == alone
    assert batched.views_that_fit(ctx, 8, 15, "cuda", image_bytes=200 * GIB) == 1
    assert scatter_solver.free_memory("cuda") == 108 * GIB
