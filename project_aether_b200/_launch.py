"""Device and stream of a call, with little host time: a small call's kernels take less time
than looking these up through `torch.cuda.device` and `torch.cuda.current_stream`."""

import contextlib

import torch

_SAME_DEVICE = contextlib.nullcontext()


def on_device(device: torch.device):
    """Context in which `device` is the current CUDA device."""
    if device.index is None or torch.cuda.current_device() == device.index:
        return _SAME_DEVICE
    return torch.cuda.device(device)


def device_index(device: torch.device) -> int:
    """Number of a CUDA device; `cuda` without one is the current device."""
    return torch.cuda.current_device() if device.index is None else device.index


def raw_stream(device: torch.device) -> int:
    """Handle of PyTorch's current stream on `device`."""
    index = device.index
    return torch._C._cuda_getCurrentRawStream(torch.cuda.current_device() if index is None else index)
