"""What sorts a group of a settled state: teams, blocks, sparse groups, dense groups in the general path's finish kernel, wide
and large buckets in the tail kernel.  At the edges of their capacities, against the CPU oracle, bit for bit."""

import pytest
import torch

import project_aether_b200 as pa
from project_aether_b200 import particle_sort
import test_settled_sort_gpu
from test_settled_sort_gpu import LARGE, LEAST, _crowd, _dt, _run, _sorted_state, _words

pytestmark = pytest.mark.gpu

# Words of the workspace header; the second: groups of dense spans, wider than a team's.
TEAM_GROUPS, WIDE_GROUPS, LARGE_BUCKETS, WIDE_BUCKETS = 54, 55, 56, 57
TEAM_TARGET = 104                                     # records of a team's bucket, on average at most


@pytest.mark.parametrize('records,wide,large', [(511, 0, 0), (512, 0, 0), (513, 1, 0), (4095, 1, 0), (4096, 1, 0),
                                                (4097, 1, 1)])
def test_a_bucket_at_a_capacity(cuda, records, wide, large):
    """One bucket has exactly `records`, most of them in one cell; nothing moves."""
    n, cells = LEAST + 100, (64, 64, 64)
    grid, pos, vel = _sorted_state(n, cells, cuda, 31)
    vel.zero_()
    shift = max(s for s in range(7) if n <= TEAM_TARGET * (64 ** 3 >> s))
    here = n // 2
    bucket = sum((pos[k][here].item() * cells[k] / grid.hi[k]) // 1 * 64 ** k for k in range(3)) // 2 ** shift
    own = [(p * (c / h)).floor() for p, c, h in zip(pos, cells, grid.hi)]
    in_bucket = ((own[0] + 64 * own[1] + 4096 * own[2]) // 2 ** shift == bucket).nonzero().flatten()
    first, last = in_bucket[0].item(), in_bucket[-1].item()
    assert last - first + 1 == in_bucket.numel() < records
    _crowd(pos, vel, first, records)  # so many from the bucket's first on
    _run(grid, pos, vel, _dt(grid), cuda, 'settled')
    words = _words(cuda)
    assert words[LARGE] == wide and words[LARGE_BUCKETS] == large and (words[WIDE_GROUPS] > 0) == wide
    assert words[TEAM_GROUPS] > 0


# Sparse grids and full cells (blocks), either side of the lower line between teams and blocks.  (The upper one is below.)
@pytest.mark.parametrize('n,cells', [(LEAST + 7, (96, 100, 90)), (LEAST + 1, (66, 66, 66)), (LEAST + 1, (64, 66, 66)),
                                     (2_000_003, (17, 17, 18)), (2_000_003, (17, 17, 17)), (2_100_001, (13, 13, 13))])
def test_sparse_and_full_cells(cuda, n, cells):
    grid, pos, vel = _sorted_state(n, cells, cuda, 32)
    _run(grid, pos, vel, _dt(grid), cuda, 'settled')


@pytest.mark.parametrize('off', [(1, 0), (0, 2), (3, 3)])
@pytest.mark.parametrize('squeeze', [None, (0.3, 0.01)])
def test_outputs_off_16_byte_boundaries(cuda, off, squeeze):
    """`off`: elements by which positions, and keys and indices, start behind a boundary."""
    n = LEAST + 3
    grid, pos, vel = _sorted_state(n, (64, 64, 64), cuda, 33, squeeze=squeeze)
    plain = pa.sort_and_gather_particles(*pos, vel, grid, 1)
    move = lambda t, k: torch.cat([t.new_zeros(k), t])[k:]
    order = plain.order._replace(keys=move(plain.order.keys, off[1]), particle_index=move(plain.order.particle_index, off[1]))
    out = particle_sort.SortedParticles(order, tuple(move(t, off[0]) for t in plain.positions), plain.velocity)
    _run(grid, pos, vel, _dt(grid), cuda, 'settled', out=out)


def _bucket_of(n, cells, records, device, drop=0):
    """A state with one bucket of exactly `records`, most of them in one cell; nothing moves."""
    grid, pos, vel = _sorted_state(n, cells, device, 31, drop=drop)
    vel.zero_()
    total = cells[0] * cells[1] * cells[2]
    shift = max(s for s in range(7) if n <= TEAM_TARGET * (total >> s))
    own = [(p * (c / h)).floor().clamp(max=c - 1) for p, c, h in zip(pos, cells, grid.hi)]
    bucket = ((own[0] + cells[0] * (own[1] + cells[1] * own[2])) // 2 ** shift)
    first = (bucket == bucket[n // 2]).nonzero()[0].item()
    _crowd(pos, vel, first, records)
    return grid, pos, vel


@pytest.mark.parametrize('drop', [0, 1])
@pytest.mark.parametrize('records,wide', [(2047, 0), (2048, 0), (2049, 1)])
def test_a_bucket_at_the_capacity_of_a_dense_group(cuda, records, wide, drop):
    grid, pos, vel = _bucket_of(LEAST + 100, (64, 64, 64), records, cuda, drop)
    _run(grid, pos, vel, _dt(grid), cuda, 'settled')
    words = _words(cuda)
    assert words[WIDE_GROUPS] > 0 and words[WIDE_BUCKETS] == wide and words[LARGE_BUCKETS] == 0


# Layers of other widths, small and large blocks of the general path's finish kernel, aligned and not.
@pytest.mark.parametrize('n,cells,squeeze,drop', [(LEAST + 2, (60, 64, 61), (0.5, 0.05), 0), (LEAST + 5, (60, 64, 61), (0.5, 0.05), 3),
                                                  (2_500_001, (29, 29, 29), (0.28, 0.03), 1), (2_500_001, (29, 29, 29), (0.5, 0.1), 0),
                                                  (40_000_001, (170, 170, 170), (0.5, 0.05), 0),
                                                  (40_000_003, (170, 170, 170), (0.2, 0.02), 1)])
def test_dense_spans(cuda, n, cells, squeeze, drop):
    grid, pos, vel = _sorted_state(n, cells, cuda, 34, squeeze=squeeze, drop=drop)
    _run(grid, pos, vel, _dt(grid), cuda, 'settled')
    words = _words(cuda)
    assert words[TEAM_GROUPS] > 0 and words[WIDE_GROUPS] > 1


def test_what_lies_near_a_dense_layer_stays_with_the_teams(cuda):
    """A tenth of the particles in a layer one cell thick: four of five particles at least are sorted by teams, 512 places each."""
    n = 4_000_000
    grid, pos, vel = _sorted_state(n, (79, 79, 79), cuda, 35, squeeze=(0.1, 0.01))
    _run(grid, pos, vel, _dt(grid), cuda, 'settled')
    words = _words(cuda)
    assert words[WIDE_GROUPS] > 0 and words[TEAM_GROUPS].item() * 512 > 0.8 * n


def test_a_counter_that_wraps_in_a_dense_group(cuda):
    """300 particles with equal shuffle bits meet in a cell of some 800: the dense group gives the call to the digit passes."""
    test_settled_sort_gpu.test_counters_that_wrap(cuda, 800, 'settled')


# Either side of the line below which grids are sparse, with and without dense layers; the fewest particles to a cell that such a call has.
@pytest.mark.parametrize('n,cells,squeeze,drop', [(1_600_000, (128, 125, 128), None, 0), (1_600_001, (128, 125, 128), None, 1),
                                                  (LEAST, (160, 160, 160), (0.3, 0.1), 2), (LEAST + 1, (160, 160, 160), (0.1, 0.01), 0),
                                                  (LEAST + 3, (200, 160, 131), (0.7, 0.02), 3), ((1 << 24) + 3, (322, 322, 322), (0.5, 0.3), 1)])
def test_sparse_grids(cuda, n, cells, squeeze, drop):
    grid, pos, vel = _sorted_state(n, cells, cuda, 36, squeeze=squeeze, drop=drop)
    _run(grid, pos, vel, _dt(grid), cuda, 'settled')
    assert _words(cuda)[TEAM_GROUPS] >= n // 512


def test_groups_of_a_sparse_grid_are_short(cuda):
    """By a block of 512 threads with four records each, groups of some 400 records, 1.6 M particles in 160^3 cells took more than
    without such groups."""
    n = 1_600_000
    grid, pos, vel = _sorted_state(n, (160, 160, 160), cuda, 37)
    push = (_dt(grid), grid.lo, grid.hi)
    out = pa.sort_and_gather_particles(*pos, vel, grid, 1, push=push)

    def took(share):
        times = []
        for _ in range(6):
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            begin.record()
            for k in range(5):
                pa.sort_and_gather_particles(*pos, vel, grid, k, push=(_dt(grid, share), grid.lo, grid.hi), out=out)
            end.record()
            torch.cuda.synchronize()
            times.append(begin.elapsed_time(end) / 5)
        return min(times)

    settled, given_up = took(0.021), took(1.0)
    assert settled < 0.85 * given_up, (settled, given_up)


# The upper line between teams and blocks, 384 to a cell: groups of one cell each, or of five.
@pytest.mark.parametrize('n,teams', [(384 * 5202, True), (384 * 5202 + 1, False)])
def test_full_cells_either_side_of_the_line(cuda, n, teams):
    grid, pos, vel = _sorted_state(n, (17, 17, 18), cuda, 38)
    _run(grid, pos, vel, _dt(grid), cuda, 'settled')
    words = _words(cuda)
    assert words[WIDE_GROUPS] == 0 and words[LARGE] == 0
    assert words[TEAM_GROUPS] == 5202 if teams else words[TEAM_GROUPS] < 5202 // 4


@pytest.mark.parametrize('drop', [0, 1])
def test_full_cells_of_teams_some_above_their_capacity(cuda, drop):
    """Half of the space with some 465 to a cell, the other with 307: cells above 512 here and there."""
    grid, pos, vel = _sorted_state(384 * 5202 - 4, (17, 17, 18), cuda, 39, squeeze=(0.205, 0.5), drop=drop)
    _run(grid, pos, vel, _dt(grid), cuda, 'settled')
    words = _words(cuda)
    assert words[TEAM_GROUPS] > 2000 and words[WIDE_GROUPS] > 10 and words[WIDE_BUCKETS] == 0


# More buckets above all shapes' capacities than the tail kernel has blocks: of several cells, and of one.
@pytest.mark.parametrize('drop', [0, 1])
@pytest.mark.parametrize('n,cells,squeeze', [(LEAST + 4, (64, 63, 64), (0.72, 0.01)), (2_000_000, (16, 63, 16), (0.58, 0.01))])
def test_many_buckets_that_no_block_holds(cuda, n, cells, squeeze, drop):
    grid, pos, vel = _sorted_state(n, cells, cuda, 40, squeeze=squeeze, drop=drop)
    _run(grid, pos, vel, _dt(grid, 0.002), cuda, 'settled')
    blocks = torch.cuda.get_device_properties(cuda).multi_processor_count
    assert _words(cuda)[LARGE_BUCKETS] > blocks
