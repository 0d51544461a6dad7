"""The sort of a moved state that starts cell-sorted: the settled path and the conditions under
which it gives the call to the general path.  Against the CPU oracle, bit for bit."""

import numpy as np
import pytest
import torch

import project_aether_b200 as pa
from oracle import sort_oracle as so
from project_aether_b200 import particle_sort

pytestmark = pytest.mark.gpu

LEAST = 3 << 19  # particles from which on the settled path is tried: while slots are reserved tile by tile
LEAST_UNTILED = 1 << 24
SETTLE_FAILED, LARGE, GROUPS = 12, 13, 54  # words of the workspace header


def _words(device):
    torch.cuda.synchronize()
    workspace = particle_sort._workspaces[(device.index, torch.cuda.current_stream(device).cuda_stream)]
    return workspace[:256].view(torch.int32).cpu()


def _route(device):
    """'settled', 'given up', or 'general' where the settled path was not tried."""
    words = _words(device)
    if words[SETTLE_FAILED]:
        return 'given up'
    return 'settled' if words[GROUPS] or words[LARGE] else 'general'  # digit passes clear the first


def _sorted_state(n, cells, device, seed, squeeze=None, drift=0.0, drop=0):
    """A state in cell order.  `squeeze`: (share, width) of particles pressed into a thin y-layer.
    `drop`: leading elements cut off, so that the arrays start off 16-byte boundaries."""
    grid = pa.CellGrid((0., 0., 0.), (1., 1., 0.7), cells)
    gen = torch.Generator(device=device).manual_seed(seed)
    n += drop
    x, y, z = (torch.rand(n, device=device, generator=gen) for _ in range(3))
    z *= 0.7
    if squeeze:
        layer = torch.rand(n, device=device, generator=gen) < squeeze[0]
        y[layer] = 0.5 + squeeze[1] * (y[layer] - 0.5)
    vel = torch.zeros((3, -(-n // 4) * 4), device=device)
    vel[:, :n] = torch.randn((3, n), device=device, generator=gen)
    vel[0, :n] += drift
    state = pa.sort_and_gather_particles(x, y, z, vel, grid, seed)
    velocity = state.velocity[:, drop:n] if drop else state.velocity
    return grid, [t[drop:] for t in state.positions], velocity


def _oracle(grid, pos, vel, n, dt, seed, **slab):
    p = [np.ascontiguousarray(t.cpu().numpy()) for t in pos]
    v = np.ascontiguousarray(vel.cpu().numpy())
    p, rows = so.push_particles(p, [v[k, :n] for k in range(3)], dt, grid.lo, grid.hi)
    v[:, :n] = np.stack(rows)
    return so.c_sort_particles(*[np.ascontiguousarray(a) for a in p], v,
                               so.Grid(grid.lo, grid.hi, grid.cells), seed, **slab)


def _check(got, want, n):
    order, *payload = want
    np.testing.assert_array_equal(got.order.keys.cpu().numpy().view(np.uint32), order.keys)
    np.testing.assert_array_equal(got.order.particle_index.cpu().numpy(), order.particle_index)
    np.testing.assert_array_equal(got.order.cell_counts.cpu().numpy(), order.cell_counts)
    np.testing.assert_array_equal(got.order.cell_start.cpu().numpy(), order.cell_start)
    for g, w in zip(got.positions, payload):
        np.testing.assert_array_equal(g.cpu().numpy(), w)
    np.testing.assert_array_equal(got.velocity.cpu().numpy()[:, :n], payload[3][:, :n])


def _crowd(pos, vel, first, count):
    """Puts `count` particles from `first` on in one place, where they stay."""
    for t in pos:
        t[first:first + count] = t[first].item()
    vel[:, first:first + count] = 0.0


def _run(grid, pos, vel, dt, device, route, out=None, digits=False, slab={}):
    n, seed = pos[0].numel(), 0x9876543210 + pos[0].numel()
    want = _oracle(grid, pos, vel, n, dt, seed, **slab)
    got = pa.sort_and_gather_particles(*pos, vel, grid, seed, push=(dt, grid.lo, grid.hi), out=out, **slab)
    assert pa.last_sort_status(device) == 0
    assert pa.last_sort_used_digit_passes(device) == digits
    assert _route(device) == route
    _check(got, want, n)


def _dt(grid, share=0.021):
    return share / max(c / h for c, h in zip(grid.cells, grid.hi))


# The smallest sizes, odd ones, sparse and full cells, cells of a bucket's size and more, and buckets
# that are no multiple of the spans the tables are made in.
@pytest.mark.parametrize('n,cells,route', [(LEAST - 1, (64, 64, 64), 'general'), (LEAST, (64, 64, 64), 'settled'),
                                           (LEAST + 1, (101, 97, 89), 'settled'), (2_300_003, (33, 32, 31), 'settled'),
                                           (3_000_001, (17, 16, 15), 'settled'), (2_500_000, (13, 11, 9), 'general'),
                                           (5_000_011, (256, 128, 100), 'settled'),
                                           (6_291_457, (107, 103, 101), 'general'),
                                           (LEAST_UNTILED - 1, (128, 128, 128), 'general'),
                                           (LEAST_UNTILED + 1, (131, 127, 113), 'settled')])
def test_settled_calls(cuda, n, cells, route):
    grid, pos, vel = _sorted_state(n, cells, cuda, n)
    _run(grid, pos, vel, _dt(grid), cuda, route)


@pytest.mark.parametrize('drift,share', [(0.0, 0.0), (5.0, 0.021), (-5.0, 0.05)])
def test_no_movers_and_a_stream_against_a_wall(cuda, drift, share):
    grid, pos, vel = _sorted_state(LEAST + 77, (80, 64, 64), cuda, 3, drift=drift)
    _run(grid, pos, vel, _dt(grid, share), cuda, 'settled')


@pytest.mark.parametrize('drop', [1, 2, 3])
def test_unaligned_arrays(cuda, drop):
    grid, pos, vel = _sorted_state(LEAST + 5, (64, 64, 64), cuda, 4, drop=drop)
    _run(grid, pos, vel, _dt(grid), cuda, 'settled')


def test_dense_layer(cuda):
    grid, pos, vel = _sorted_state(4_000_000, (128, 64, 64), cuda, 5, squeeze=(0.3, 0.1))
    _run(grid, pos, vel, _dt(grid), cuda, 'settled')


def test_buckets_that_no_block_holds(cuda):
    """Most of the particles in a thin layer: most buckets there are above a team's capacity, many above a dense group's."""
    grid, pos, vel = _sorted_state(4_000_000, (128, 64, 64), cuda, 6, squeeze=(0.7, 0.02))
    _run(grid, pos, vel, _dt(grid), cuda, 'settled')


# Some buckets that no team holds (those that no block holds, in numbers: test_settled_shapes_gpu.py); unaligned arrays; cells
# above the capacity of a dense group; a mean of some 200 to a cell; blocks of the large finish shape behind.
@pytest.mark.parametrize('n,cells,squeeze,drop', [(LEAST, (64, 64, 64), (0.3, 0.002), 0),
                                                  (LEAST + 3, (101, 97, 89), (0.28, 0.03), 1),
                                                  (2_000_001, (32, 32, 32), (0.6, 0.01), 0),
                                                  (LEAST, (20, 21, 20), (0.7, 0.04), 0),
                                                  (40_000_003, (180, 170, 160), (0.28, 0.02), 0)])
def test_dense_layers_of_some_buckets(cuda, n, cells, squeeze, drop):
    grid, pos, vel = _sorted_state(n, cells, cuda, 21, squeeze=squeeze, drop=drop)
    _run(grid, pos, vel, _dt(grid), cuda, 'settled')
    assert _words(cuda)[LARGE] > 0


@pytest.mark.parametrize('crowd,digits', [(2_700, False), (5_000, False), (6_000, True)])
def test_one_cell_of_thousands(cuda, crowd, digits):
    """Blocks of the tail kernel hold 5120 records; a cell of more goes to the digit passes, as it does in
    the general path."""
    n = LEAST + 100
    grid, pos, vel = _sorted_state(n, (64, 64, 64), cuda, 10)
    _crowd(pos, vel, n // 2, crowd)
    _run(grid, pos, vel, _dt(grid), cuda, 'settled', digits=digits)
    assert _words(cuda)[LARGE] == 1

def test_too_many_movers(cuda):
    grid, pos, vel = _sorted_state(LEAST, (64, 64, 64), cuda, 7)
    _run(grid, pos, vel, _dt(grid, 1.0), cuda, 'given up')


@pytest.mark.parametrize('some,every', [(2, 7), (3, 7)])
def test_a_part_of_the_input_with_many_movers(cuda, some, every):
    """Some particles of every seven of one block of the scan leave their bucket, and hardly any other."""
    grid, pos, vel = _sorted_state(LEAST, (64, 64, 64), cuda, 14)
    dt = _dt(grid, 0.001)
    here = torch.arange(50 * 6144, 51 * 6144, device=cuda)
    here = here[here % every < some]
    vel[1, here] = (1.5 / 64 / dt) * (1 - 2 * (pos[1][here] > 0.5).float())
    _run(grid, pos, vel, dt, cuda, 'settled')


@pytest.mark.parametrize('most', [16, 30])
def test_movers_that_the_sample_does_not_see(cuda, most):
    """The sample is every 48th particle of the scan's blocks.  A third of all particles leave their bucket:
    more than there is room for in all; five of eight: more than a block's list holds."""
    grid, pos, vel = _sorted_state(LEAST, (64, 64, 64), cuda, 15)
    dt = _dt(grid, 0.001)
    at = torch.arange(LEAST, device=cuda) % 48
    here = (at >= 1) & (at <= most)
    vel[1, :LEAST][here] = (1.5 / 64 / dt) * (1 - 2 * (pos[1][here] > 0.5).float())
    _run(grid, pos, vel, dt, cuda, 'given up')


# On either side of the share from which on the general path is faster, which is another for each of its plans.
@pytest.mark.parametrize('n,cells,share,route', [(LEAST, (64, 64, 64), 0.15, 'settled'),
                                                 (LEAST, (64, 64, 64), 0.35, 'given up'),
                                                 (LEAST_UNTILED + 1, (128, 128, 128), 0.06, 'settled'),
                                                 (LEAST_UNTILED + 1, (128, 128, 128), 0.15, 'given up'),
                                                 (40_000_003, (180, 170, 160), 0.1, 'settled'),
                                                 (40_000_003, (180, 170, 160), 0.25, 'given up')])
def test_shares_of_movers(cuda, n, cells, share, route):
    """`share`: of the particles leave their cell."""
    grid, pos, vel = _sorted_state(n, cells, cuda, 16)
    _run(grid, pos, vel, _dt(grid, share / 2.39), cuda, route)

@pytest.mark.parametrize('where', [0, 777_777, -1])
def test_one_particle_out_of_order(cuda, where):
    """Two particles of far-apart buckets change places; -1: the last with the first."""
    grid, pos, vel = _sorted_state(LEAST + 3, (64, 64, 64), cuda, 8)
    other = LEAST // 2 if where >= 0 else 0
    for t in (*pos, *(vel[k] for k in range(3))):
        t[where], t[other] = t[other].item(), t[where].item()
    _run(grid, pos, vel, _dt(grid), cuda, 'given up')


def test_random_order(cuda):
    grid, pos, vel = _sorted_state(LEAST + 9, (64, 64, 64), cuda, 9)
    shuffle = torch.randperm(LEAST + 9, device=cuda)
    pos = [t[shuffle].contiguous() for t in pos]
    vel[:, :LEAST + 9] = vel[:, shuffle]
    _run(grid, pos, vel, _dt(grid), cuda, 'given up')


def test_a_crowded_cell_that_a_group_holds(cuda):
    """Every cell of a group has 32 counters: 2000 particles of one cell are some 60 on each."""
    n, crowd = LEAST + 100, 2_000
    grid, pos, vel = _sorted_state(n, (128, 128, 128), cuda, 10)
    for t in pos:
        t[n // 2:n // 2 + crowd] = t[n // 2].item()
    vel[:, n // 2:n // 2 + crowd] = 0.0
    _run(grid, pos, vel, _dt(grid), cuda, 'settled')


def _same_shuffle_bits(n, seed, first, last):
    """Particles whose keys have the same shuffle bits."""
    bits = so.shuffle_bits(n, seed)
    return first + np.flatnonzero(bits[first:last] == bits[first])


@pytest.mark.parametrize('crowd,route', [(0, 'given up'), (3_000, 'settled')])
def test_counters_that_wrap(cuda, crowd, route):
    """300 particles with equal shuffle bits meet in one cell: more than a counter of one byte counts.  Among a
    group's records the sort is given up, after other groups have been written, and done from the start; in
    a bucket of the tail kernel it goes to the digit passes."""
    n, cells = LEAST + 100, (64, 64, 64)
    grid, pos, vel = _sorted_state(n, cells, cuda, 17)
    dt, seed = _dt(grid), 0x9876543210 + n
    to = n // 2
    if crowd:
        _crowd(pos, vel, to, crowd)
    same = _same_shuffle_bits(n, seed, 1, n - 1)
    same = torch.from_numpy(same[np.linspace(0, same.size - 1, 300).astype(np.int64)]).to(cuda)
    for k, h in enumerate(cells):
        centre = ((pos[k][to] * h / grid.hi[k]).floor() + 0.5) / h * grid.hi[k]
        vel[k, same] = (centre - pos[k][same]) / dt
    _run(grid, pos, vel, dt, cuda, route, digits=True)


@pytest.mark.parametrize('ix_offset,nx_local', [(0, 33), (16, 32), (43, 21)])
@pytest.mark.parametrize('drop', [0, 1])
def test_slabs(cuda, ix_offset, nx_local, drop):
    """A state in the order of a slab's cells.  Particles that leave the slab are binned into its nearest column."""
    n, cells = LEAST + 11 + drop, (64, 60, 50)
    grid = pa.CellGrid((0., 0., 0.), (1., 1., 0.7), cells)
    gen = torch.Generator(device=cuda).manual_seed(18)
    x, y, z = (torch.rand(n, device=cuda, generator=gen) for _ in range(3))
    x = (ix_offset + x * nx_local) / cells[0]
    vel = torch.zeros((3, -(-n // 4) * 4), device=cuda)
    vel[:, :n] = torch.randn((3, n), device=cuda, generator=gen)
    slab = {'ix_offset': ix_offset, 'nx_local': nx_local}
    state = pa.sort_and_gather_particles(x, y, z * 0.7, vel, grid, 3, **slab)
    pos = [t[drop:] for t in state.positions]
    _run(grid, pos, state.velocity[:, drop:n] if drop else state.velocity, _dt(grid), cuda, 'settled', slab=slab)

def test_outputs_over_the_inputs(cuda):
    n = LEAST + 4
    grid, pos, vel = _sorted_state(n, (64, 64, 64), cuda, 11)
    spare = pa.sort_and_gather_particles(*pos, vel, grid, 1)
    out = particle_sort.SortedParticles(spare.order, tuple(pos), vel)
    _run(grid, pos, vel, _dt(grid), cuda, 'general', out=out)


def test_positions_that_are_no_numbers_and_walls_far_off(cuda):
    grid, pos, vel = _sorted_state(LEAST, (64, 64, 64), cuda, 12)
    vel[0, 1000] = float('inf')
    vel[1, 2000] = float('nan')
    vel[2, 3000] = 1e30
    _run(grid, pos, vel, _dt(grid), cuda, 'settled')


def test_capture_and_replay(cuda):
    n = LEAST + 21
    grid, pos, vel = _sorted_state(n, (64, 64, 64), cuda, 13)
    dt, seed = _dt(grid), 0x9876543210 + n
    want = _oracle(grid, pos, vel, n, dt, seed)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        out = pa.sort_and_gather_particles(*pos, vel, grid, seed, push=(dt, grid.lo, grid.hi))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        pa.sort_and_gather_particles(*pos, vel, grid, seed, push=(dt, grid.lo, grid.hi), out=out)
    for t in (*out.order, *out.positions, out.velocity):
        t.zero_()
    graph.replay()
    torch.cuda.synchronize()
    _check(out, want, n)
