"""Device and stream of a call (project_aether_b200/_launch.py)."""

import pytest
import torch

import project_aether_b200 as pa
from project_aether_b200 import _launch, particle_sort


def test_a_device_without_a_number_is_the_current_one(monkeypatch):
    monkeypatch.setattr(torch.cuda, 'current_device', lambda: 3)
    monkeypatch.setattr(torch._C, '_cuda_getCurrentRawStream', lambda index: 100 + int(index),
                        raising=False)
    assert _launch.raw_stream(torch.device('cuda')) == 103
    assert _launch.raw_stream(torch.device('cuda', 1)) == 101
    assert _launch.on_device(torch.device('cuda')) is _launch.on_device(torch.device('cuda', 3))
    # Nothing was sorted on that device and stream.
    monkeypatch.setattr(particle_sort, '_workspaces', {})
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
