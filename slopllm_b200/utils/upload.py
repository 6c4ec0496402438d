"""Small tables from the host to the device without waiting for the stream."""
from __future__ import annotations

import torch


def upload(values, dtype: torch.dtype, device) -> torch.Tensor:
    """`values` (numbers, any nesting) as a tensor on `device`.  They cross from pinned memory: a copy from pageable memory waits until all
    that the stream holds has run, and the kernels behind it are launched late.  The pinned block is the allocator's again, and is not
    handed out before the copy has read it."""
    t = torch.tensor(values, dtype=dtype)
    device = torch.device(device)
    return t.pin_memory().to(device, non_blocking=True) if device.type == "cuda" else t.to(device)
