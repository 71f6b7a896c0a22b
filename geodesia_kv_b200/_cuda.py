"""Current stream and device of a call, at the cost of a call.

``torch.cuda.current_stream`` and ``torch.cuda.device`` resolve and re-check the device on every use; a decode call
needs three of them, which together took longer than launching its kernels.
"""
from __future__ import annotations

import torch


def stream(dev: torch.device) -> int:
    """Handle of the device's current stream."""
    return torch._C._cuda_getCurrentRawStream(torch.cuda.current_device() if dev.index is None else dev.index)


class _Here:
    def __enter__(self):
        return None

    def __exit__(self, *exc):
        return False


_HERE = _Here()


def on(dev: torch.device):
    """Context in which ``dev`` is the current device; nothing is switched where it already is."""
    return _HERE if dev.index is None or dev.index == torch.cuda.current_device() else torch.cuda.device(dev)
