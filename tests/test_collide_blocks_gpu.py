"""The collision kernel where its blocks of 16 to 256 cells end, and with more pairs than threads."""

import numpy as np
import pytest
import torch

import project_aether_b200 as pa
from oracle import collide_oracle as co
from test_collide import compare_with_oracle, run_gpu


@pytest.mark.gpu
@pytest.mark.parametrize('cells', [1, 255, 256, 257, 513])
@pytest.mark.parametrize('mean,factor', [(3.0, 2.0e15), (40.0, 5.0e13)])
def test_blocks_of_cells(cuda, cells, mean, factor):
    counts = np.random.default_rng(cells).poisson(mean, cells)
    counts[-1] = 2 * (cells % 7) + 1  # an odd cell at the end of the last block
    counts[cells // 2] = 1500         # more pairs than a block has threads
    case = co.make_case(counts, rng_seed=cells, selection_factor=factor, seed=99, step=5)
    assert compare_with_oracle(case, run_gpu(case, cuda)) > 0


# Blocks of 16 cells as long as there is room for them on the multiprocessors, then of 32, ...
@pytest.mark.gpu
@pytest.mark.parametrize('cells_per_block', [16, 32, 64, 128, 256])
@pytest.mark.parametrize('more', [-1, 1])
def test_where_blocks_grow(cuda, cells_per_block, more):
    places = 6 * torch.cuda.get_device_properties(cuda).multi_processor_count
    cells = places * cells_per_block + more
    counts = np.random.default_rng(cells).poisson(2.0, cells)
    counts[[0, cells // 2, -1]] = (700, 1500, 3)
    case = co.make_case(counts, rng_seed=cells, selection_factor=2.0e15, seed=9, step=4)
    assert compare_with_oracle(case, run_gpu(case, cuda)) > 0


@pytest.mark.gpu
def test_few_dense_cells_fill_the_multiprocessors(cuda):
    """The same particles and pairs in 1000 cells and in 16,000: much the same time."""
    library = pa.ntc_collide.load_library()
    n, times = 400_000, []
    for cells in (16_000, 1000):
        velocity = torch.randn((3, n), device=cuda)
        start = (torch.arange(cells + 1, device=cuda) * (n // cells)).int()
        sigma = torch.full((cells,), 3.0, device=cuda)
        accepted = torch.zeros(cells, dtype=torch.int32, device=cuda)
        params = pa.CollisionParams(0.15 / (n / cells * 3.0), 1.7, 0.46, 5, 0)
        samples = []
        for _ in range(9):
            begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            begin.record()
            for _ in range(50):
                pa.collide(library, velocity, start, sigma, accepted, n, params)
            end.record()
            torch.cuda.synchronize()
            samples.append(begin.elapsed_time(end) / 50)
        assert 0 < int(accepted.sum())
        times.append(sorted(samples)[4])
    assert times[1] < 2.5 * times[0], times  # 256 cells to every block: 4 to 5 times
