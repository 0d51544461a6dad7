"""The kernels that work in phases, with fewer blocks than they have pieces of work: as when
something else holds multiprocessors and the other blocks cannot start.  Against the ordinary
call, bit for bit."""

import ctypes

import pytest
import torch

import project_aether_b200 as pa
from project_aether_b200 import _native
from project_aether_b200.particle_sort import native_grid

pytestmark = pytest.mark.gpu


def _few_blocks(pos, vel, grid, seed, most_blocks, payload, device):
    """(status, handed over, results) of a call whose kernels get at most `most_blocks` blocks."""
    lib = _native.load_library()
    n, cells = pos[0].numel(), grid.num_cells
    keys, index, counts, start = (torch.full((k,), -1, dtype=torch.int32, device=device)
                                  for k in (n, n, cells, cells + 1))
    xs, ys, zs = (torch.zeros(n, device=device) for _ in range(3))
    vs = torch.zeros_like(vel)
    ws = torch.empty(lib.AetherSortWorkspaceBytes(n, cells, 1), dtype=torch.uint8, device=device)
    sorted_arrays = [t.data_ptr() if payload else None for t in (xs, ys, zs, vs)]
    stream = torch.cuda.current_stream(device).cuda_stream
    _native.check(lib.AetherSortProbeFewBlocks(
        *(t.data_ptr() for t in pos), vel.data_ptr() if payload else None, vel.shape[1], n,
        ctypes.byref(native_grid(grid)), seed, keys.data_ptr(), index.data_ptr(),
        counts.data_ptr(), start.data_ptr(), *sorted_arrays, vel.shape[1], most_blocks,
        ws.data_ptr(), ws.numel(), stream), 'AetherSortProbeFewBlocks')
    status, used = ctypes.c_int32(-1), ctypes.c_int32(-1)
    _native.check(lib.AetherSortReadStatus(ws.data_ptr(), stream, ctypes.byref(status)), 'status')
    _native.check(lib.AetherSortReadUsedDigitPasses(ws.data_ptr(), stream, ctypes.byref(used)), 'used')
    payload_out = (xs, ys, zs, vs) if payload else ()
    return status.value, bool(used.value), (keys, index, counts, start, *payload_out)


# Even; a layer whose buckets a block has to cut; a cell that only the digit passes can take.
# One launch (one, a dozen, all 296 tiles), and the kernel behind the finish of a middling call.
@pytest.mark.parametrize('most_blocks', [1, 2, 5, 100])
@pytest.mark.parametrize('n,edge', [(300, 4), (5_000, 16), (606_208, 48), (900_001, 48)])
@pytest.mark.parametrize('density', ['even', 'layer', 'cell'])
def test_any_number_of_blocks_finishes_the_call(cuda, n, edge, density, most_blocks):
    grid = pa.CellGrid((0., 0., 0.), (1., 1., 1.), (edge,) * 3)
    gen = torch.Generator(device=cuda).manual_seed(n)
    pos = [torch.rand(n, device=cuda, generator=gen) for _ in range(3)]
    vel = torch.zeros((3, -(-n // 4) * 4), device=cuda)
    vel[:, :n] = torch.randn((3, n), device=cuda, generator=gen)
    if density == 'layer':
        pos[2][: n // 2] = 0.51
    elif density == 'cell':
        for p in pos:
            p[: n // 2] = 0.51
    want = pa.sort_and_gather_particles(*pos, vel, grid, 99)
    for payload in (True, False):
        status, handed_over, got = _few_blocks(pos, vel, grid, 99, most_blocks, payload, cuda)
        assert status == 0
        assert handed_over == (density == 'cell' and n > 100_000)
        for g, w in zip(got, (*want.order, *want.positions, want.velocity)):
            assert torch.equal(g, w)


# Groups without payload whose byte counters wrap, finished again bucket by bucket.
@pytest.mark.parametrize('most_blocks', [1, 7])
@pytest.mark.parametrize('n,edge,crowd', [(200_003, 96, 4_600), (2_400_011, 128, 3_000)])
def test_any_number_of_blocks_finishes_wrapped_groups(cuda, n, edge, crowd, most_blocks):
    grid = pa.CellGrid((0., 0., 0.), (1., 1., 1.), (edge,) * 3)
    gen = torch.Generator(device=cuda).manual_seed(n)
    pos = [torch.rand(n, device=cuda, generator=gen) for _ in range(3)]
    for p in pos:
        p[:crowd] = 0.251
        p[crowd:2 * crowd] = 0.751
    vel = torch.zeros((3, n), device=cuda)
    want = pa.sort_particles_by_cell(*pos, grid, 99)
    status, handed_over, got = _few_blocks(pos, vel, grid, 99, most_blocks, False, cuda)
    assert (status, handed_over) == (0, False)
    for g, w in zip(got, want):
        assert torch.equal(g, w)


# One launch, and the kernel behind the finish of a middling call.
@pytest.mark.parametrize('n', [5_000, 600_000, 1_200_000])
@pytest.mark.parametrize('kept', [1, 120])
def test_a_call_does_not_wait_for_a_kernel_beside_it(cuda, n, kept):
    """A kernel of another stream keeps the shared memory of one multiprocessor, or of most, for
    200 ms: a part of the call's blocks runs, and does the work of the others."""
    lib = _native.load_library()
    grid = pa.CellGrid((0., 0., 0.), (1., 1., 1.), (32, 32, 32))
    pos = [torch.rand(n, device=cuda) for _ in range(3)]
    vel = torch.randn((3, n), device=cuda)
    beside, stream = torch.cuda.Stream(cuda), torch.cuda.Stream(cuda)
    scratch = torch.empty(8192, dtype=torch.uint8, device=cuda)
    returned = torch.zeros(1, dtype=torch.int32, device=cuda)
    with torch.cuda.stream(stream):  # the workspace and the arrays of the call below exist
        want = pa.sort_and_gather_particles(*pos, vel, grid, 3)
        arrays = pa.sort_and_gather_particles(*pos, vel, grid, 4)
    torch.cuda.synchronize()
    _native.check(lib.AetherSortProbeWaitGiveUp(scratch.data_ptr(), scratch.numel(), kept, 200 * 1024,
                                                200_000_000, returned.data_ptr(), beside.cuda_stream),
                  'AetherSortProbeWaitGiveUp')
    ended = torch.cuda.Event()
    ended.record(beside)
    with torch.cuda.stream(stream):
        got = pa.sort_and_gather_particles(*pos, vel, grid, 3, out=arrays)
        stream.synchronize()
    assert not ended.query(), 'the call waited for the kernel beside it'
    torch.cuda.synchronize()
    assert int(returned) == kept
    for g, w in zip((*got.order, *got.positions, got.velocity),
                    (*want.order, *want.positions, want.velocity)):
        assert torch.equal(g, w)
