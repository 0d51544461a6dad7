"""The padding columns of the sorted velocities become zero, whatever kernel does it."""

import pytest
import torch

import project_aether_b200 as pa
from project_aether_b200 import particle_sort

pytestmark = pytest.mark.gpu

GRID = pa.CellGrid((0., 0., 0.), (1., 1., 1.), (12, 11, 10))


def _state(device, n):
    gen = torch.Generator(device=device).manual_seed(n)
    pos = tuple(torch.rand(n, device=device, generator=gen) for _ in range(3))
    return pos, torch.randn((3, n), device=device, generator=gen)


# One launch, tiles, digit passes; columns for a few, many, and none.
@pytest.mark.parametrize('n,path', [(1, 0), (5001, 0), (5001, 1), (700_001, 0), (2_000_003, 0)])
@pytest.mark.parametrize('extra', [0, 1, 70_000])
@pytest.mark.parametrize('given', [False, True])
@pytest.mark.parametrize('push', [None, (1e-3, (0., 0., 0.), (1., 1., 1.))])
def test_columns_behind_the_particles(cuda, n, path, extra, given, push):
    pos, vel = _state(cuda, n)
    plain = pa.sort_and_gather_particles(*pos, vel, GRID, 9, path=path, push=push)
    out = None
    if given:
        out = particle_sort.SortedParticles(plain.order, plain.positions, torch.full((3, n + extra), 7., device=cuda))
        version = out.velocity._version
    got = pa.sort_and_gather_particles(*pos, vel, GRID, 9, path=path, push=push, padded_out=n + extra, out=out)
    assert got.velocity.shape == (3, n + extra)
    assert torch.equal(got.velocity[:, :n], plain.velocity) and not got.velocity[:, n:].any()
    if given and extra:
        assert out.velocity._version > version


@pytest.mark.parametrize('n', [5001, 700_001])
def test_padding_over_an_input(cuda, n):
    """The columns become zero before anything is read."""
    pos, vel = _state(cuda, n)
    buffer = torch.empty(3 * (2 * n + 4), device=cuda)
    velocity = buffer.view(3, 2 * n + 4)
    x = velocity[0, n:2 * n]
    x.copy_(pos[0])
    plain = pa.sort_and_gather_particles(torch.zeros_like(pos[0]), *pos[1:], vel, GRID, 9)
    out = particle_sort.SortedParticles(plain.order._replace(keys=plain.order.keys.clone()),
                                        tuple(t.clone() for t in plain.positions), velocity)
    got = pa.sort_and_gather_particles(x, *pos[1:], vel, GRID, 9, padded_out=2 * n + 4, out=out)
    assert torch.equal(got.order.keys, plain.order.keys) and torch.equal(got.velocity[:, :n], plain.velocity)
    assert not got.velocity[:, n:].any()


def test_an_output_that_wants_gradients_is_refused(cuda):
    pos, vel = _state(cuda, 5001)
    plain = pa.sort_and_gather_particles(*pos, vel, GRID, 9)
    wants = torch.zeros((3, 5004), device=cuda, requires_grad=True)
    out = particle_sort.SortedParticles(plain.order, plain.positions, wants)
    with pytest.raises(RuntimeError):
        pa.sort_and_gather_particles(*pos, vel, GRID, 9, padded_out=5004, out=out)


@pytest.mark.parametrize('n', [5001, 700_001])
def test_wide_padding_is_zeroed_by_all_multiprocessors(cuda, n):
    """Room for 8 M particles more is 96 MB of zeros: 2.3 ms through two blocks, some 50 us through all."""
    extra = 8_000_000
    pos, vel = _state(cuda, n)
    out = pa.sort_and_gather_particles(*pos, vel, GRID, 9, padded_out=n + extra)
    out.velocity.fill_(7.)
    took = []
    for _ in range(5):
        begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        begin.record()
        pa.sort_and_gather_particles(*pos, vel, GRID, 9, padded_out=n + extra, out=out)
        end.record()
        torch.cuda.synchronize()
        took.append(begin.elapsed_time(end))
    assert not out.velocity[:, n:].any()
    assert min(took) < 1.0


@pytest.mark.parametrize('n,path', [(0, 0), (5001, 0), (5001, 1)])
def test_rows_of_more_than_2_to_the_31_bytes(cuda, n, path):
    """A row of the sorted velocities may be longer than the largest pitch of a 2D copy."""
    pos, vel = _state(cuda, n + 1)
    plain = pa.sort_and_gather_particles(*(p[:n] for p in pos), vel, GRID, 9, path=path)
    rows = torch.full((3, (1 << 29) + 8), 7., device=cuda)
    out = particle_sort.SortedParticles(plain.order, plain.positions, rows)
    got = pa.sort_and_gather_particles(*(p[:n] for p in pos), vel, GRID, 9, path=path, padded_out=rows.shape[1], out=out)
    assert torch.equal(got.velocity[:, :n], plain.velocity[:, :n])
    assert not any(row[n:].any() for row in got.velocity)
