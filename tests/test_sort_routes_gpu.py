"""The sort at the edges of its routes: the one-launch sort of small calls, tiles of the scatter
kernels, parts of the scans, 8-byte records of calls without payload.  Against the CPU oracle,
bit for bit."""

import numpy as np
import pytest
import torch

import project_aether_b200 as pa
from oracle import sort_oracle as so
from project_aether_b200 import workloads

pytestmark = pytest.mark.gpu


def _state(n, device, seed, drift=0.0):
    gen = torch.Generator(device=device).manual_seed(seed)
    pos = [torch.rand(n, device=device, generator=gen) for _ in range(3)]
    vel = torch.zeros((3, -(-n // 4) * 4), device=device)
    vel[:, :n] = torch.randn((3, n), device=device, generator=gen) + drift
    return pos, vel


def _compare(n, cells, device, moved, squeeze=None, drop=0):
    """`squeeze`: (share, width) of particles pressed into a thin y-layer.  `drop`: leading
    elements cut off, so that the arrays start off 16-byte boundaries."""
    grid = pa.CellGrid((0., 0., 0.), (1., 1., 1.), cells)
    pos, vel = _state(n + drop, device, n)
    if squeeze:
        share, width = squeeze
        layer = torch.rand(n + drop, device=device,
                           generator=torch.Generator(device=device).manual_seed(5)) < share
        pos[1][layer] = 0.5 + width * (pos[1][layer] - 0.5)
    pos = [t[drop:] for t in pos]
    vel = vel[:, drop:n + drop] if drop else vel
    seed, dt = 0x123456789 + n, 3e-3
    got = pa.sort_and_gather_particles(*pos, vel, grid, seed,
                                       push=(dt, grid.lo, grid.hi) if moved else None)
    assert pa.last_sort_status(device) == 0
    assert not pa.last_sort_used_digit_passes(device)
    order = pa.sort_particles_by_cell(*(got.positions if moved else pos), grid, seed)
    assert pa.last_sort_status(device) == 0
    assert not pa.last_sort_used_digit_passes(device)
    p = [np.ascontiguousarray(t.cpu().numpy()) for t in pos]
    v = np.ascontiguousarray(vel.cpu().numpy())
    if moved:
        p, rows = so.push_particles(p, [v[k, :n] for k in range(3)], dt, grid.lo, grid.hi)
        v[:, :n] = np.stack(rows)
        p = [np.ascontiguousarray(a) for a in p]
    ogrid = so.Grid(grid.lo, grid.hi, grid.cells)
    want, *payload = so.c_sort_particles(*p, v, ogrid, seed)
    results = [(got.order, want)]
    if moved:  # the sorted, moved particles again, without payload: input in cell order
        again = so.c_sort_particles(*[np.ascontiguousarray(t.cpu().numpy()) for t in got.positions],
                                    v, ogrid, seed)[0]
        results.append((order, again))
    else:
        results.append((order, want))
    for g, w in results:
        np.testing.assert_array_equal(g.keys.cpu().numpy().view(np.uint32), w.keys)
        np.testing.assert_array_equal(g.particle_index.cpu().numpy(), w.particle_index)
        np.testing.assert_array_equal(g.cell_counts.cpu().numpy(), w.cell_counts)
        np.testing.assert_array_equal(g.cell_start.cpu().numpy(), w.cell_start)
    for g, w in zip(got.positions, payload):
        np.testing.assert_array_equal(g.cpu().numpy(), w)
    np.testing.assert_array_equal(got.velocity.cpu().numpy()[:, :n], payload[3][:, :n])


# A tile is 512 to 2048 particles; 148 multiprocessors with two blocks each take 606,208.
@pytest.mark.parametrize('n,cells', [(1, (1, 1, 1)), (511, (3, 5, 7)), (512, (64, 64, 64)),
                                     (513, (25, 25, 16)), (2_049, (100, 100, 100)),
                                     (151_553, (32, 32, 16)), (606_207, (64, 64, 32)),
                                     (606_208, (13, 11, 9)), (606_209, (64, 64, 32))])
@pytest.mark.parametrize('moved', [False, True])
def test_small_calls(cuda, n, cells, moved):
    _compare(n, cells, cuda, moved)


# Slots reserved tile by tile; rows of counts that are no multiple of four and pass into a second
# part of the scan; tiles of the split that are cut; a plan with more buckets than the split takes.
@pytest.mark.parametrize('n,cells', [(700_001, (128, 64, 64)), (1_212_417, (64, 64, 64)),
                                     (2_500_003, (25, 25, 16)), (6_291_457, (97, 89, 83)),
                                     (5_000_001, (331, 257, 211))])
@pytest.mark.parametrize('moved', [False, True])
def test_middling_calls(cuda, n, cells, moved):
    _compare(n, cells, cuda, moved)


# Tiles of 512 and of 1024 threads, with four buckets per thread of the split and with some more.
@pytest.mark.parametrize('n,cells', [(700_001, (128, 128, 128)), (700_001, (128, 128, 129)),
                                     (2_500_003, (256, 128, 128)), (2_500_003, (256, 128, 129))])
def test_buckets_per_thread_of_the_split(cuda, n, cells):
    _compare(n, cells, cuda, False)


@pytest.mark.parametrize('n,cells', [(300_000, (64, 32, 32)), (3_000_000, (64, 64, 64))])
def test_dense_layers_and_unaligned_arrays(cuda, n, cells):
    _compare(n, cells, cuda, False, squeeze=(0.7, 0.03))
    _compare(n, cells, cuda, False, drop=1)


def test_counters_of_sixteen_bits_are_emptied_in_time(cuda):
    """Above 51,200 buckets the counts are kept in 16 bits.  A crowded bucket, its particles side
    by side in memory, takes one block's counter past 2^15 several times."""
    n, crowd = 218_000_000, 120_000
    grid = pa.CellGrid((0., 0., 0.), (1., 1., 1.), (512, 256, 256))
    gen = torch.Generator(device=cuda).manual_seed(3)
    x, y, z = (torch.rand(n, device=cuda, generator=gen) for _ in range(3))
    at = 100_000_001
    # The 512 cells of one row are one bucket: about 240 particles a cell.
    x[at:at + crowd] = torch.rand(crowd, device=cuda, generator=gen)
    y[at:at + crowd] = 0.5004
    z[at:at + crowd] = 0.2504
    vel = torch.zeros((3, n), device=cuda)
    got = pa.sort_and_gather_particles(x, y, z, vel, grid, 77)
    assert pa.last_sort_status(cuda) == 0
    assert not pa.last_sort_used_digit_passes(cuda)
    cell = torch.zeros(n, dtype=torch.int64, device=cuda)
    for c, cells in ((z, 256), (y, 256), (x, 512)):
        cell = cell * cells + (c * cells).to(torch.int64).clamp_(0, cells - 1)
    assert torch.equal(got.order.cell_counts.long(), torch.bincount(cell, minlength=grid.num_cells))
    keys = got.order.keys.long() & 0xFFFFFFFF
    index = got.order.particle_index.long()
    assert torch.equal(keys >> 7, cell[index])
    step = keys[1:] - keys[:-1]
    assert bool(((step > 0) | ((step == 0) & (index[1:] > index[:-1]))).all())
    assert torch.equal(got.positions[0], x[index])


# One launch; middling; large enough for the plain scatter.
@pytest.mark.parametrize('n', [40_000, 1_500_000, 7_000_000])
def test_capture_and_replay(cuda, n):
    grid = pa.CellGrid((0., 0., 0.), (1., 1., 1.), (64, 64, 32))
    pos, vel = _state(n, cuda, 8)
    other, other_vel = _state(n, cuda, 9)
    stream = torch.cuda.Stream(cuda)
    with torch.cuda.stream(stream):  # the stream's workspace exists before the capture
        pa.sort_and_gather_particles(*pos, vel, grid, 5)
        pa.sort_particles_by_cell(*pos, grid, 5)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        got = pa.sort_and_gather_particles(*pos, vel, grid, 5)
        order = pa.sort_particles_by_cell(*pos, grid, 5)
    for a, b in ((pos, vel), (other, other_vel)):
        for to, source in zip(pos, a):
            to.copy_(source)
        vel.copy_(b)
        graph.replay()
        torch.cuda.synchronize()
        want = pa.sort_and_gather_particles(*pos, vel, grid, 5)
        for g, w in zip((*got.order, *got.positions, got.velocity),
                        (*want.order, *want.positions, want.velocity)):
            assert torch.equal(g, w)
        for g, w in zip(order, want.order):
            assert torch.equal(g, w)


def test_two_streams_side_by_side(cuda):
    grid = pa.CellGrid((0., 0., 0.), (1., 1., 1.), (64, 64, 32))
    sizes = (50_000, 300_000, 1_500_000)
    states = [_state(n, cuda, n) for n in sizes]
    want = [pa.sort_and_gather_particles(*pos, vel, grid, 3) for pos, vel in states]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(cuda) for _ in range(2)]
    results = []
    for _ in range(4):
        for k, (pos, vel) in enumerate(states):
            for s in streams:
                with torch.cuda.stream(s):
                    results.append((k, pa.sort_and_gather_particles(*pos, vel, grid, 3)))
    torch.cuda.synchronize()
    for k, got in results:
        for g, w in zip((*got.order, *got.positions), (*want[k].order, *want[k].positions)):
            assert torch.equal(g, w)
