"""The collision kernel is set up while the kernel before it ends: whatever that kernel is, its results are waited for."""

import pytest
import torch

import project_aether_b200 as pa
from project_aether_b200 import ntc_collide

pytestmark = pytest.mark.gpu

CELLS, N = 4000, 64_000
PARAMS = pa.CollisionParams(0.02, 1.7, 0.46, 99, 3)


def _state(device):
    gen = torch.Generator(device=device).manual_seed(5)
    velocity = torch.randn((3, N), device=device, generator=gen)
    cell = torch.randint(0, CELLS, (N,), device=device, generator=gen)
    start = torch.zeros(CELLS + 1, dtype=torch.int32, device=device)
    start[1:] = torch.cumsum(torch.bincount(cell, minlength=CELLS), 0)
    return velocity, start, torch.full((CELLS,), 4.0, device=device)


def _collide(velocity, start, sigma):
    accepted = torch.zeros(CELLS, dtype=torch.int32, device=velocity.device)
    pa.collide(ntc_collide.load_library(), velocity, start, sigma, accepted, N, PARAMS)
    return velocity, sigma, accepted


def _want(device):
    state = _state(device)
    torch.cuda.synchronize()
    want = _collide(*state)
    torch.cuda.synchronize()
    assert want[2].sum() > 0
    return want


def _late(state, out):
    """Fills `out` from `state` behind work that takes a while, in the kernels right before the collisions."""
    big = torch.ones(1 << 26, device=out[0].device)
    for _ in range(4):
        big.mul_(1.5)
    for o, s in zip(out, state):
        o.copy_(s + (big[:1] * 0).to(s.dtype))


@pytest.mark.parametrize('other_stream', [False, True])
def test_behind_kernels_of_others(cuda, other_stream):
    want, state = _want(cuda), _state(cuda)
    out = [torch.zeros_like(t) for t in state]
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    if other_stream:
        with torch.cuda.stream(side):
            _late(state, out)
        torch.cuda.current_stream().wait_stream(side)
    else:
        _late(state, out)
    got = _collide(*out)
    assert all(torch.equal(g, w) for g, w in zip(got, want))


def test_captured_behind_another_stream(cuda):
    want, state = _want(cuda), _state(cuda)
    out = [torch.zeros_like(t) for t in state]
    accepted = torch.zeros(CELLS, dtype=torch.int32, device=cuda)
    library = ntc_collide.load_library()
    torch.cuda.synchronize()
    main, side, graph = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=main):
        side.wait_stream(main)
        with torch.cuda.stream(side):
            for o, s in zip(out, state):
                o.copy_(s)
        main.wait_stream(side)
        pa.collide(library, *out, accepted, N, PARAMS)
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(g, w) for g, w in zip((*out[:1], out[2], accepted), want))


# Kernels that let the collisions in before they end: the sort in one launch does so when all its blocks run, and writes on.
# `crowd`: in one cell, so many that the call ends in the digit passes, behind that point.
@pytest.mark.parametrize('n,crowd', [(5001, 0), (20_003, 6000), (100_003, 0), (200_003, 6000), (500_001, 0), (500_001, 6000)])
@pytest.mark.parametrize('captured', [False, True])
def test_behind_a_sort_in_one_launch(cuda, n, crowd, captured):
    grid = pa.CellGrid((0., 0., 0.), (1., 1., 1.), (20, 20, 10))
    gen = torch.Generator(device=cuda).manual_seed(n)
    pos = [torch.rand(n, device=cuda, generator=gen) for _ in range(3)]
    for t in pos:
        t[:crowd] = 0.5
    vel = torch.randn((3, n), device=cuda, generator=gen)
    library = ntc_collide.load_library()
    sigma, accepted = torch.empty(CELLS, device=cuda), torch.empty(CELLS, dtype=torch.int32, device=cuda)
    stream = torch.cuda.Stream()

    def step(out, between):
        out = pa.sort_and_gather_particles(*pos, vel, grid, 5, padded_out=-(-n // 4) * 4, out=out)
        between()
        pa.collide(library, out.velocity, out.order.cell_start, sigma, accepted, n, PARAMS)
        return out

    def outputs(out):
        return [t.clone() for t in (*out.order, *out.positions, out.velocity, sigma, accepted)]

    with torch.cuda.stream(stream):
        sigma.fill_(4.0)
        out = step(None, torch.cuda.synchronize)
        want = outputs(out)
        assert pa.last_sort_used_digit_passes(cuda) == bool(crowd) and want[-1].sum() > 0
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    if captured:
        with torch.cuda.graph(graph, stream=stream):
            step(out, lambda: None)
    for _ in range(5):
        with torch.cuda.stream(stream):
            for t in (*out.order, *out.positions, out.velocity):
                t.zero_()
            sigma.fill_(4.0)
            graph.replay() if captured else step(out, lambda: None)
            got = outputs(out)
        torch.cuda.synchronize()
        assert all(torch.equal(g, w) for g, w in zip(got, want))
