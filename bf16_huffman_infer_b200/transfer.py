"""Layers between host and device memory at the rate of the link.

A checkpoint's tensors and the compressed buffers a conversion hands back are ordinary (pageable) host memory.  The
driver moves such memory through one staging buffer with one thread: on B200 over PCIe 5, 32 MB take 1.8 ms to the
device and 15.6 ms back into a new tensor, most of it page faults, where the link itself needs 0.6 ms.  Here the data
goes through a few page-locked slabs, filled or emptied by all of torch's intra-op threads while the copy engine works
on the next one.  The slabs come from torch's caching host allocator (at most ``SLABS`` of ``SLAB_BYTES`` per running
call, given back to it at the end), so nothing is kept here and calls from several threads or streams do not meet.
"""
from __future__ import annotations

from typing import Callable, Optional

import torch
from torch import Tensor

# Two slabs of 8 MB: 32 MB take 0.99 ms up and 1.8 ms down (4 MB: 1.12 / 2.3, 2 MB: 1.19 / 4.1; a third or fourth slab
# changes nothing).  What is left of the way down is page faults of the new tensor.
SLAB_BYTES = 8 << 20
SLABS = 2
_SMALL = 1 << 20             # below this one plain copy is as fast


def _slabs(nbytes: int):
    count = min(SLABS, -(-nbytes // SLAB_BYTES))
    return [torch.empty(SLAB_BYTES, dtype=torch.uint8, device="cpu", pin_memory=True) for _ in range(count)]


def upload_rows(src: Tensor, dst: Tensor, arrived: Optional[Callable[[int, int], None]] = None) -> None:
    """Copies a host matrix into a device matrix of its shape on the device's current stream.  ``arrived(lo, hi)`` is
    called when the copy of rows ``lo..hi-1`` has been enqueued: what it launches there overlaps the rest of the copy."""
    rows, row_bytes = src.shape[0], src.shape[1] * src.element_size()
    stream = torch.cuda.current_stream(dst.device)
    step = max(1, SLAB_BYTES // row_bytes)
    if src.is_pinned() or rows * row_bytes <= _SMALL or row_bytes > SLAB_BYTES:
        dst.copy_(src, non_blocking=src.is_pinned())
        if arrived is not None:
            arrived(0, rows)
        if src.is_pinned():
            stream.synchronize()              # the caller may change or drop the source
        return
    slabs = _slabs(rows * row_bytes)
    views = [s[:step * row_bytes].view(src.dtype).view(step, src.shape[1]) for s in slabs]
    sent = [torch.cuda.Event() for _ in slabs]
    for i, lo in enumerate(range(0, rows, step)):
        hi, at = min(rows, lo + step), i % len(slabs)
        if i >= len(slabs):
            sent[at].synchronize()
        view = views[at][:hi - lo]
        view.copy_(src[lo:hi])
        dst[lo:hi].copy_(view, non_blocking=True)
        sent[at].record(stream)
        if arrived is not None:
            arrived(lo, hi)


def download(src: Tensor, out: Optional[Tensor] = None) -> Tensor:
    """A device tensor as a host tensor (``out``, contiguous and pageable, or a new one); complete when the call returns."""
    nbytes = src.numel() * src.element_size()
    if nbytes <= _SMALL:
        return src.cpu() if out is None else out.copy_(src)
    stream = torch.cuda.current_stream(src.device)
    if out is None:
        out = torch.empty(src.shape, dtype=src.dtype, device="cpu")
    flat_src, flat_out = src.contiguous().view(-1).view(torch.uint8), out.view(-1).view(torch.uint8)
    slabs = _slabs(nbytes)
    here = [torch.cuda.Event() for _ in slabs]
    spans = [(lo, min(nbytes, lo + SLAB_BYTES)) for lo in range(0, nbytes, SLAB_BYTES)]

    def fetch(i: int) -> None:
        lo, hi = spans[i]
        slabs[i % len(slabs)][:hi - lo].copy_(flat_src[lo:hi], non_blocking=True)
        here[i % len(slabs)].record(stream)

    for i in range(min(len(slabs), len(spans))):
        fetch(i)
    for i, (lo, hi) in enumerate(spans):
        here[i % len(slabs)].synchronize()
        flat_out[lo:hi].copy_(slabs[i % len(slabs)][:hi - lo])
        if i + len(slabs) < len(spans):
            fetch(i + len(slabs))
    return out
