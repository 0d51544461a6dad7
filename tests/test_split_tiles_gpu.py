"""Calls without payload: tiles of the split at the sizes where their length, the rounds or the kernel change, and either
side of one chunk of records.  Against the CPU oracle, bit for bit."""

import numpy as np
import pytest
import torch

import project_aether_b200 as pa
from oracle import sort_oracle as so

pytestmark = pytest.mark.gpu


def _sizes():
    """(tiles of 512 x 4, 8, 16 particles for all blocks, and one more or less), (rounds that are not whole)."""
    for rounds, per_block in ((1, 2048), (1, 4096), (1, 8192), (2, 8192), (3, 8192)):
        for more in (-1, 0, 1):
            yield rounds, per_block, more


@pytest.mark.parametrize('drop', [0, 1])
@pytest.mark.parametrize('rounds,per_block,more', list(_sizes()))
def test_around_whole_rounds(cuda, rounds, per_block, more, drop):
    blocks = 2 * torch.cuda.get_device_properties(cuda).multi_processor_count
    _check(cuda, rounds * per_block * blocks + more, (40, 41, 39), drop)


@pytest.mark.parametrize('n,cells', [(1 << 24, (64, 64, 64)), ((1 << 24) + 1, (64, 64, 64)), ((1 << 24) - 3, (128, 128, 128)),
                                     (3_000_001, (7, 7, 7)), (2_500_003, (130, 128, 128))])
def test_chunk_edges_and_few_or_many_buckets(cuda, n, cells):
    _check(cuda, n, cells, 0)


def _check(cuda, n, cells, drop):
    grid = pa.CellGrid((0., 0., 0.), (1., 1., 1.), cells)
    gen = torch.Generator(device=cuda).manual_seed(n)
    pos = [torch.rand(n + drop, device=cuda, generator=gen)[drop:] for _ in range(3)]
    got = pa.sort_particles_by_cell(*pos, grid, 77)
    assert pa.last_sort_status(cuda) == 0 and not pa.last_sort_used_digit_passes(cuda)
    want, *_ = so.c_sort_particles(*[np.ascontiguousarray(t.cpu().numpy()) for t in pos], None,
                                   so.Grid(grid.lo, grid.hi, grid.cells), 77)
    np.testing.assert_array_equal(got.keys.cpu().numpy().view(np.uint32), want.keys)
    np.testing.assert_array_equal(got.particle_index.cpu().numpy(), want.particle_index)
    np.testing.assert_array_equal(got.cell_start.cpu().numpy(), want.cell_start)
    np.testing.assert_array_equal(got.cell_counts.cpu().numpy(), want.cell_counts)
