"""The collision kernel where its blocks of 256 cells end, and with more pairs than threads."""

import numpy as np
import pytest

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
