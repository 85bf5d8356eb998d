"""Small host-side helpers shared by the ops (counterpart of flash_moe/ops/utils.py)."""

from __future__ import annotations

import torch
from torch.autograd import forward_ad


def contiguous(t):
    """The reference makes every tensor argument contiguous before a kernel sees it (ops/utils.py:35-45)."""
    return t.contiguous() if isinstance(t, torch.Tensor) else t


_grad_enabled, _tracing = torch.is_grad_enabled, torch._C._is_tracing


def plain_call() -> bool:
    """True where an op may run without its autograd node, which costs several microseconds of host time: no gradient is
    recorded, no forward-mode level is open (the node is what refuses tangents, which would be dropped silently) and
    torch.jit is not tracing (the node is what a trace records)."""
    return not _grad_enabled() and forward_ad._current_level < 0 and not _tracing()
