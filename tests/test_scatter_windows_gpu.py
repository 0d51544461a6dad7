"""Above 2^26 particles input in random order is scattered window by window, input in some order as below.
Just above the line, with and without payload, against the CPU oracle, bit for bit."""

import numpy as np
import pytest
import torch

import project_aether_b200 as pa
from oracle import sort_oracle as so
from project_aether_b200 import particle_sort

pytestmark = pytest.mark.gpu

N = (1 << 26) + 5
SHARED_ROUNDS = 15  # word of the workspace header


@pytest.mark.parametrize('payload', [True, False])
@pytest.mark.parametrize('ordered', [False, True])
def test_either_kernel(cuda, ordered, payload):
    cells = (128, 128, 128) if payload else (257, 256, 256)  # without payload: more buckets than a split takes
    grid = pa.CellGrid((0., 0., 0.), (1., 1., 1.), cells)
    gen = torch.Generator(device=cuda).manual_seed(41)
    x, y, z = (torch.rand(N, device=cuda, generator=gen) for _ in range(3))
    vel = torch.zeros((3, -(-N // 4) * 4), device=cuda)
    vel[:, :N] = torch.randn((3, N), device=cuda, generator=gen)
    if ordered:
        state = pa.sort_and_gather_particles(x, y, z, vel, grid, 3)
        (x, y, z), vel = state.positions, state.velocity
    seed = 0x1122334455
    if payload:
        got = pa.sort_and_gather_particles(x, y, z, vel, grid, seed)
        order = got.order
    else:
        order = pa.sort_particles_by_cell(x, y, z, grid, seed)
    assert pa.last_sort_status(cuda) == 0 and not pa.last_sort_used_digit_passes(cuda)
    torch.cuda.synchronize()
    workspace = particle_sort._workspaces[(cuda.index, torch.cuda.current_stream(cuda).cuda_stream)]
    # Of the count kernel's rounds, 2048 particles each with so many buckets, nearly all or hardly any: the line is half of them.
    shared, rounds = workspace[:256].view(torch.int32)[SHARED_ROUNDS].item(), N // 2048
    assert 0.9 * rounds < shared <= rounds + 1000 if ordered else shared < 0.1 * rounds
    host = [np.ascontiguousarray(t.cpu().numpy()) for t in (x, y, z)]
    want, *rest = so.c_sort_particles(*host, np.ascontiguousarray(vel.cpu().numpy()),
                                      so.Grid(grid.lo, grid.hi, grid.cells), seed)
    np.testing.assert_array_equal(order.keys.cpu().numpy().view(np.uint32), want.keys)
    np.testing.assert_array_equal(order.particle_index.cpu().numpy(), want.particle_index)
    np.testing.assert_array_equal(order.cell_start.cpu().numpy(), want.cell_start)
    if payload:
        for g, w in zip(got.positions, rest):
            np.testing.assert_array_equal(g.cpu().numpy(), w)
        np.testing.assert_array_equal(got.velocity.cpu().numpy()[:, :N], rest[3][:, :N])
