"""Device and stream of a call, with little host time: a small call's kernels take less time
than looking these up through `torch.cuda.device` and `torch.cuda.current_stream`."""

import contextlib

import torch

_SAME_DEVICE = contextlib.nullcontext()


def on_device(device: torch.device):
    """Context in which `device` is the current CUDA device."""
    if torch.cuda.current_device() == device.index:
        return _SAME_DEVICE
    return torch.cuda.device(device)


def numbered(device: torch.device) -> torch.device:
    """The device by its number; `cuda` without one is the current device."""
    return torch.device('cuda', torch.cuda.current_device()) if device.index is None else device


def raw_stream(device: torch.device) -> int:
    """Handle of PyTorch's current stream on `device`, which has a number."""
    return torch._C._cuda_getCurrentRawStream(device.index)
