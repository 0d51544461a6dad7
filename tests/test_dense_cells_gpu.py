"""Cells of tens to thousands of particles: the finish kernels' counters are then divided by index.
Against the CPU oracle, bit for bit."""

import numpy as np
import pytest
import torch

import project_aether_b200 as pa
from oracle import sort_oracle as so

pytestmark = pytest.mark.gpu


def _check(n, cells, device, in_order):
    grid = pa.CellGrid((0., 0., 0.), (1., 1., 1.), cells)
    gen = torch.Generator(device=device).manual_seed(n)
    pos = [torch.rand(n, device=device, generator=gen) for _ in range(3)]
    vel = torch.randn((3, n), device=device, generator=gen)
    if in_order:  # all particles of a cell side by side: their indices agree in the highest bits
        order = pa.sort_particles_by_cell(*pos, grid, 1).particle_index.long()
        pos = [t[order] for t in pos]
    seed = 0x77 + n
    got = pa.sort_and_gather_particles(*pos, vel, grid, seed)
    assert pa.last_sort_status(device) == 0 and not pa.last_sort_used_digit_passes(device)
    keys_only = pa.sort_particles_by_cell(*pos, grid, seed)
    assert pa.last_sort_status(device) == 0 and not pa.last_sort_used_digit_passes(device)
    want, *payload = so.c_sort_particles(*[t.cpu().numpy() for t in pos], vel.cpu().numpy(),
                                         so.Grid(grid.lo, grid.hi, grid.cells), seed)
    for g in (got.order, keys_only):
        np.testing.assert_array_equal(g.keys.cpu().numpy().view(np.uint32), want.keys)
        np.testing.assert_array_equal(g.particle_index.cpu().numpy(), want.particle_index)
        np.testing.assert_array_equal(g.cell_counts.cpu().numpy(), want.cell_counts)
        np.testing.assert_array_equal(g.cell_start.cpu().numpy(), want.cell_start)
    for g, w in zip((*got.positions, got.velocity), payload):
        np.testing.assert_array_equal(g.cpu().numpy(), w)


# Fewer particles than the index bits a counter could take; one cell; sizes about a power of two (a bit
# of the index more or less); every route (one launch, tiles, buckets, large blocks).
@pytest.mark.parametrize('n,cells', [(1, (1, 1, 1)), (3, (1, 1, 1)), (127, (2, 1, 1)), (1_024, (1, 1, 1)),
                                     (1_025, (1, 1, 1)), (2_560, (2, 1, 1)), (5_120, (3, 1, 1)), (65_536, (5, 5, 5)),
                                     (65_537, (5, 5, 5)), (400_000, (10, 10, 10)), (606_209, (12, 12, 12)),
                                     (1_300_001, (25, 25, 25)), (4_000_000, (25, 25, 16)), (8_388_609, (40, 40, 40)),
                                     (37_000_003, (30, 30, 30))])
@pytest.mark.parametrize('in_order', [False, True])
def test_dense_cells(cuda, n, cells, in_order):
    _check(n, cells, cuda, in_order)
