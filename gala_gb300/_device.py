"""Device plumbing: torch tensors as the owners of device memory and streams."""
from __future__ import annotations

import numpy as np
import torch


def require_cuda() -> torch.device:
    if not torch.cuda.is_available():
        raise RuntimeError("gala_gb300 needs a CUDA device: no GPU is visible to torch")
    return torch.device("cuda", torch.cuda.current_device())


def stream_handle(stream=None) -> int:
    s = stream if stream is not None else torch.cuda.current_stream()
    return int(s.cuda_stream)


def as_device_f64(a, device=None) -> torch.Tensor:
    """Contiguous float64 CUDA tensor view/copy of ``a`` (numpy, list or tensor)."""
    dev = device or require_cuda()
    if isinstance(a, torch.Tensor):
        # a pinned host tensor is copied asynchronously on the current stream
        nb = a.device.type == "cpu" and a.is_pinned()
        return a.to(device=dev, dtype=torch.float64, non_blocking=nb).contiguous()
    arr = np.ascontiguousarray(np.asarray(a, dtype=np.float64))
    if not arr.flags.writeable:
        arr = arr.copy()
    return torch.from_numpy(arr).to(dev)


def ptr(t: torch.Tensor) -> int:
    return int(t.data_ptr())


# Host arrays up to this many values go through one page-locked block that the
# kernel reads and writes in place: no allocation, copy and wait on either side of
# the launch.  Both sides of the line in the docstring below.
STAGED_VALUES = 1 << 15


def call_staged(name, head, a, out_size):
    """One evaluation entry point ``name(*head, a, n, out, stream)`` on the host array
    ``a`` (rows, n): the result's ``out_size`` values as a new numpy array.

    The block comes from torch's page-locked cache and goes back to it when the
    stream has been waited for.  Measured on a GB300, potential gradient of an MW
    composite, device copies / in place: 257 points 95 / 50 us, 5,000 96 / 70 us,
    10,900 96 / 88 us, 40,000 105 / 180 us."""
    from . import _abi

    size = a.size
    block = torch.empty(size + out_size, dtype=torch.float64, pin_memory=True)
    host = block.numpy()
    host[:size].reshape(a.shape)[...] = a
    p = block.data_ptr()
    s = torch.cuda.current_stream()
    try:
        _abi.call(name, *head, p, a.shape[1], p + 8 * size, int(s.cuda_stream))
    finally:  # the block is not given back before the kernel is done with it
        s.synchronize()
    return host[size:].copy()
