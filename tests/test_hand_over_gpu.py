"""Calls that the bucketed path hands over to the digit passes on the device, where one kernel
then runs them all, and calls that it keeps although they are crowded."""

import numpy as np
import pytest
import torch

import project_aether_b200 as pa
from oracle import sort_oracle as so

pytestmark = pytest.mark.gpu


def _state(n, device, seed):
    gen = torch.Generator(device=device).manual_seed(seed)
    pos = [torch.rand(n, device=device, generator=gen) for _ in range(3)]
    vel = torch.zeros((3, -(-n // 4) * 4), device=device)
    vel[:, :n] = torch.randn((3, n), device=device, generator=gen)
    return pos, vel


# One, two, three and four passes (key widths of 8, 10, 22 and 28 bits); tiles of 6144 keys cut
# exactly, one short and one over, and more tiles than multiprocessors.
@pytest.mark.parametrize('n,cells', [(6_144, (2, 1, 1)), (12_287, (7, 1, 1)), (40_001, (32, 32, 32)),
                                     (6_145, (128, 128, 128)), (1_200_007, (64, 64, 128))])
@pytest.mark.parametrize('moved', [False, True])
def test_dense_cell_is_sorted_by_the_digit_passes(cuda, n, cells, moved):
    grid = pa.CellGrid((0., 0., 0.), (1., 1., 1.), cells)
    pos, vel = _state(n, cuda, n)
    crowd = torch.arange(n, device=cuda) % 7 != 0  # most particles in one cell
    for k in range(3):
        pos[k][crowd] = 0.4
        vel[k, :n][crowd] *= 1e-6
    dt = 1e-3
    push = (dt, grid.lo, grid.hi) if moved else None
    seed = 0x1234567 + n
    got = pa.sort_and_gather_particles(*pos, vel, grid, seed, push=push)
    assert pa.last_sort_status(cuda) == 0
    assert pa.last_sort_used_digit_passes(cuda)
    p = [t.cpu().numpy() for t in pos]
    v = vel.cpu().numpy()
    if moved:
        p, rows = so.push_particles(p, [v[k, :n] for k in range(3)], dt, grid.lo, grid.hi)
        v[:, :n] = np.stack(rows)
    want = so.sort_particles(*p, so.Grid(grid.lo, grid.hi, grid.cells), seed)
    sorted_payload = so.gather_payload(want.particle_index, *p, v)
    np.testing.assert_array_equal(got.order.keys.cpu().numpy().view(np.uint32), want.keys)
    np.testing.assert_array_equal(got.order.particle_index.cpu().numpy(), want.particle_index)
    np.testing.assert_array_equal(got.order.cell_counts.cpu().numpy(), want.cell_counts)
    np.testing.assert_array_equal(got.order.cell_start.cpu().numpy(), want.cell_start)
    for g, w in zip((*got.positions, got.velocity), sorted_payload):
        np.testing.assert_array_equal(g.cpu().numpy(), w)
    # The same particles without payload.
    order = pa.sort_particles_by_cell(*(torch.from_numpy(np.ascontiguousarray(a)).to(cuda) for a in p),
                                      grid, seed)
    assert pa.last_sort_status(cuda) == 0
    assert pa.last_sort_used_digit_passes(cuda)
    np.testing.assert_array_equal(order.keys.cpu().numpy().view(np.uint32), want.keys)
    np.testing.assert_array_equal(order.particle_index.cpu().numpy(), want.particle_index)
    np.testing.assert_array_equal(order.cell_counts.cpu().numpy(), want.cell_counts)
    np.testing.assert_array_equal(order.cell_start.cpu().numpy(), want.cell_start)


def _sorted_as_by_the_oracle(pos, vel, grid, seed, cuda):
    got = pa.sort_and_gather_particles(*pos, vel, grid, seed)
    assert pa.last_sort_status(cuda) == 0
    handed_over = pa.last_sort_used_digit_passes(cuda)
    want, *payload = so.c_sort_particles(*(t.cpu().numpy() for t in pos), vel.cpu().numpy(),
                                         so.Grid(grid.lo, grid.hi, grid.cells), seed)
    order = pa.sort_particles_by_cell(*pos, grid, seed)
    assert pa.last_sort_status(cuda) == 0
    for result in (got.order, order):
        np.testing.assert_array_equal(result.keys.cpu().numpy().view(np.uint32), want.keys)
        np.testing.assert_array_equal(result.particle_index.cpu().numpy(), want.particle_index)
        np.testing.assert_array_equal(result.cell_counts.cpu().numpy(), want.cell_counts)
        np.testing.assert_array_equal(result.cell_start.cpu().numpy(), want.cell_start)
    n = pos[0].numel()
    for g, w in zip(got.positions, payload):
        np.testing.assert_array_equal(g.cpu().numpy(), w)
    np.testing.assert_array_equal(got.velocity.cpu().numpy()[:, :n], payload[3][:, :n])
    return handed_over, pa.last_sort_used_digit_passes(cuda)


def _crowd(pos, chosen, cells, edge, device):
    """Puts the chosen particles, in equal parts, into the middle of `cells` cells of a cubic
    grid with `edge` cells along an axis, spread over the whole grid."""
    k = int(chosen.sum())
    cell = (torch.arange(k, device=device) % cells) * (edge ** 3 // cells)
    for axis, stride in enumerate((1, edge, edge * edge)):
        pos[axis][chosen] = ((cell // stride % edge).float() + 0.5) / edge


# Every block of a full grid finds cells that its shared memory cannot hold, or byte counters
# that wrap, at about the same time: the hand-over is decided while other blocks start, sort and
# wait.  One launch; behind the finish kernel of middling calls.
@pytest.mark.parametrize('n,edge,cells', [(500_009, 64, 60), (2_400_011, 64, 250)])
def test_many_blocks_decide_on_the_hand_over_together(cuda, n, edge, cells):
    grid = pa.CellGrid((0., 0., 0.), (1., 1., 1.), (edge,) * 3)
    for repeat in range(3):
        # Cells of 6,700 particles, more than any block holds.
        pos, vel = _state(n, cuda, n + repeat)
        _crowd(pos, torch.arange(n, device=cuda) % 6 != 0, cells, edge, cuda)
        assert _sorted_as_by_the_oracle(pos, vel, grid, 5 + repeat, cuda) == (True, True)
        # Cells of 600 particles, all of them with the same shuffle value.
        pos, vel = _state(n, cuda, n + repeat)
        seed = 77 + repeat
        same = torch.from_numpy(so.shuffle_bits(n, seed) == 9).to(cuda)
        _crowd(pos, same, int(same.sum()) // 600, edge, cuda)
        assert _sorted_as_by_the_oracle(pos, vel, grid, seed, cuda) == (True, True)


# In a grid of one particle per cell a bucket of a call without payload spans 1024 cells, on 16
# byte counters each: one cell of some 3500 records or more wraps one of them.  One launch; a
# bucket too large for a group; a group.  The bucket is then finished in runs of fewer cells.
@pytest.mark.parametrize('n,edge,crowd', [(200_003, 96, 4_600), (900_001, 128, 5_120), (2_400_011, 128, 3_900)])
def test_dense_cells_of_a_sparse_grid_stay_off_the_digit_passes(cuda, n, edge, crowd):
    grid = pa.CellGrid((0., 0., 0.), (1., 1., 1.), (edge,) * 3)
    pos, vel = _state(n, cuda, n)
    # Three cells in different buckets; the particles that fell into them before move one cell on.
    middle = (torch.floor(torch.tensor([0.2, 0.5, 0.8], device=cuda) * edge) + 0.5) / edge
    chosen = torch.arange(n, device=cuda) < 3 * crowd
    there = torch.zeros(n, dtype=torch.bool, device=cuda)
    for m in middle:
        there |= sum(((p * edge).long() == (m * edge).long()).long() for p in pos) == 3
    pos[0][there] += 1.0 / edge
    for p in pos:
        p[chosen] = middle[torch.arange(3 * crowd, device=cuda) % 3]
    order = pa.sort_particles_by_cell(*pos, grid, 11)
    assert pa.last_sort_status(cuda) == 0
    assert not pa.last_sort_used_digit_passes(cuda)
    assert int(order.cell_counts.max()) == crowd
    want = so.c_sort_particles(*(t.cpu().numpy() for t in pos), vel.cpu().numpy(),
                               so.Grid(grid.lo, grid.hi, grid.cells), 11)[0]
    np.testing.assert_array_equal(order.keys.cpu().numpy().view(np.uint32), want.keys)
    np.testing.assert_array_equal(order.particle_index.cpu().numpy(), want.particle_index)
    np.testing.assert_array_equal(order.cell_counts.cpu().numpy(), want.cell_counts)
    np.testing.assert_array_equal(order.cell_start.cpu().numpy(), want.cell_start)


# The one-launch sort with payload: cells between what a block holds with payload (2560) and what
# the bucketed path takes (5120), and a row of cells, one bucket, of 100,000 particles.
@pytest.mark.parametrize('n', [60_000, 300_000, 606_208])
@pytest.mark.parametrize('crowd', [2_561, 5_120, 'row'])
@pytest.mark.parametrize('moved', [False, True])
def test_small_calls_take_what_larger_calls_take(cuda, n, crowd, moved):
    if crowd == 'row' and n < 300_000:
        pytest.skip('fewer particles than the row has')
    grid = pa.CellGrid((0., 0., 0.), (1., 1., 1.), (64, 32, 32))
    pos, vel = _state(n, cuda, n)
    pos[2] *= 30 / 32  # the topmost layers hold the crowd alone
    if crowd == 'row':
        chosen = torch.arange(n, device=cuda) % (n // 100_000) == 0
        chosen &= torch.cumsum(chosen, 0) <= 100_000
    else:
        chosen = torch.arange(n, device=cuda) < crowd
        pos[0][chosen] = 32.5 / 64
    pos[1][chosen] = 16.5 / 32
    pos[2][chosen] = 31.5 / 32
    for k in range(3):
        vel[k, :n][chosen] *= 1e-7
    seed, dt = 31, 1e-3
    got = pa.sort_and_gather_particles(*pos, vel, grid, seed,
                                       push=(dt, grid.lo, grid.hi) if moved else None)
    assert pa.last_sort_status(cuda) == 0
    assert not pa.last_sort_used_digit_passes(cuda)
    p, v = [t.cpu().numpy() for t in pos], vel.cpu().numpy()
    if moved:
        p, rows = so.push_particles(p, [v[k, :n] for k in range(3)], dt, grid.lo, grid.hi)
        v[:, :n] = np.stack(rows)
        p = [np.ascontiguousarray(a) for a in p]
    want, *payload = so.c_sort_particles(*p, v, so.Grid(grid.lo, grid.hi, grid.cells), seed)
    np.testing.assert_array_equal(got.order.keys.cpu().numpy().view(np.uint32), want.keys)
    np.testing.assert_array_equal(got.order.particle_index.cpu().numpy(), want.particle_index)
    np.testing.assert_array_equal(got.order.cell_counts.cpu().numpy(), want.cell_counts)
    np.testing.assert_array_equal(got.order.cell_start.cpu().numpy(), want.cell_start)
    for g, w in zip(got.positions, payload):
        np.testing.assert_array_equal(g.cpu().numpy(), w)
    np.testing.assert_array_equal(got.velocity.cpu().numpy()[:, :n], payload[3][:, :n])
    if crowd != 'row':
        assert int(got.order.cell_counts.max()) == crowd
