"""Device and stream of a call (project_aether_b200/_launch.py)."""

import threading

import pytest
import torch

import project_aether_b200 as pa
from project_aether_b200 import _launch, particle_sort


def test_a_device_without_a_number_is_the_current_one(monkeypatch):
    monkeypatch.setattr(torch.cuda, 'current_device', lambda: 3)
    monkeypatch.setattr(torch._C, '_cuda_getCurrentRawStream', lambda index: 100 + int(index),
                        raising=False)
    assert _launch.numbered(torch.device('cuda')) == torch.device('cuda', 3)
    assert _launch.numbered(torch.device('cuda', 1)) == torch.device('cuda', 1)
    assert _launch.raw_stream(torch.device('cuda', 1)) == 101
    # Nothing was sorted on that device and stream.
    monkeypatch.setattr(particle_sort, '_workspaces', {})
    assert pa.last_sort_status() == 0
    assert pa.last_sort_status(torch.device('cuda')) == 0
    assert pa.last_sort_used_digit_passes(torch.device('cuda')) is False


@pytest.mark.gpu
def test_status_of_a_device_without_a_number(cuda):
    grid = pa.CellGrid((0., 0., 0.), (1., 1., 1.), (8, 8, 8))
    x, y, z = (torch.full((6_000,), 0.5, device=cuda) for _ in range(3))
    pa.sort_particles_by_cell(x, y, z, grid, 1)
    assert pa.last_sort_status(torch.device('cuda')) == 0
    assert pa.last_sort_used_digit_passes(torch.device('cuda')) == pa.last_sort_used_digit_passes(cuda)
    assert pa.last_sort_used_digit_passes(torch.device('cuda')) is True


@pytest.mark.gpu
@pytest.mark.parametrize('sizes', [((2_500_000, (25, 25, 16)), (2_600_000, (16, 16, 11))),
                                   ((16_500_000, (128, 128, 128)), (17_500_000, (128, 128, 128)))])
def test_threads_with_calls_of_different_sizes(cuda, sizes):
    """Kernels whose shared memory depends on the call, launched by two threads at a time: no
    call's setting may take the other's launch its memory away."""
    failures, results = [], [None, None]
    inputs = [[torch.rand(n, device=cuda) for _ in range(3)] for n, _ in sizes]
    grids = [pa.CellGrid((0., 0., 0.), (1., 1., 1.), cells) for _, cells in sizes]
    want = [pa.sort_particles_by_cell(*x, g, 5) for x, g in zip(inputs, grids)]
    torch.cuda.synchronize()
    calls = 4000 if sizes[0][0] < 10**7 else 400

    def work(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream(cuda)):
                for i in range(calls):
                    results[k] = pa.sort_particles_by_cell(*inputs[k], grids[k], 5)
                    if i % 50 == 49:
                        torch.cuda.current_stream().synchronize()
        except RuntimeError as error:
            failures.append(str(error))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failures
    for got, w in zip(results, want):
        for a, b in zip(got, w):
            assert torch.equal(a, b)
