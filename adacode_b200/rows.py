"""Copies of dense token rows (a token's keys and values appended to the residual, the not yet packed tails behind the
segments) and what every launch needs of the device: its current stream, its being the current one."""
from __future__ import annotations

import contextlib
import ctypes
from typing import Optional, Sequence

import torch
from torch.autograd import forward_ad
from torch.autograd.graph import increment_version

from . import _lib

_is_wrapped = torch._C._functorch.is_functorch_wrapped_tensor
_BF16 = torch.bfloat16
_HERE = contextlib.nullcontext()


def stream_ptr(device: torch.device) -> int:
    """Handle of the device's current stream."""
    index = device.index
    return torch._C._cuda_getCurrentRawStream(torch.cuda.current_device() if index is None else index)


def on_device(device: torch.device):
    """``torch.cuda.device(device)``, which costs as much as a launch, only where another device is current."""
    index = device.index
    return _HERE if index is None or index == torch.cuda.current_device() else torch.cuda.device(device)


def row_record(src: torch.Tensor, dst: torch.Tensor, rows: Optional[int] = None, at: int = 0) -> Optional[tuple]:
    """``dst[:, :, at: at + rows].copy_(src[:, :, :rows])`` (all of both without ``rows``) as a record of the row-copy
    kernel, or None if it is not one: it takes plain bf16 CUDA tensors [B, H, T, D] on one device, rows on 16-byte
    boundaries, and nothing that ``copy_`` would do beyond moving bytes: no gradient or tangent to carry on, no
    ``torch.func`` wrapper, nothing to refuse."""
    if type(src) is not torch.Tensor or type(dst) is not torch.Tensor:
        return None
    if src.dtype is not _BF16 or dst.dtype is not _BF16 or not src.is_cuda or src.get_device() != dst.get_device():
        return None
    if forward_ad._current_level >= 0 or _is_wrapped(src) or _is_wrapped(dst):
        return None
    if (src.requires_grad or dst.requires_grad) and torch.is_grad_enabled():
        return None
    if dst.is_inference() and not torch.is_inference_mode_enabled():
        return None
    from_strides, to_strides = src.stride(), dst.stride()
    if len(from_strides) != 4 or len(to_strides) != 4:
        return None
    a, b, c, u = from_strides
    d, e, f, v = to_strides
    B, H, T, D = src.shape
    B2, H2, T2, D2 = dst.shape
    if rows is None:
        rows = T if T == T2 else -1
    if B != B2 or H != H2 or D != D2 or not 0 <= rows <= T or at + rows > T2:
        return None
    from_ptr, to_ptr = src.data_ptr(), dst.data_ptr() + 2 * at * f
    if u != 1 or v != 1 or (a | b | c | d | e | f | D) & 7 or (from_ptr | to_ptr) & 15 or B * H * rows * D >= 2 ** 31:
        return None
    return (from_ptr, to_ptr, a, b, c, d, e, f, B, H, rows, D)


def copy_rows(pairs: Sequence[tuple]) -> None:
    """``dst.copy_(src)`` for every ``(src, dst)`` pair, in one launch where the kernel takes all of them.

    The caches do not use it: describing two one-token tensors costs more on the host than the launch it saves
    (keys and values of a token appended: 21.5 us, two ``copy_`` calls 19.5 us)."""
    pairs = [(s, d) for s, d in pairs if d.numel()]
    if not pairs:
        return
    dev = pairs[0][1].device
    records = [row_record(s, d) for s, d in pairs]
    for i, (s, d) in enumerate(pairs):
        # what copy_ refuses: destinations that overlap themselves or their source
        if records[i] is not None and (0 in d.stride() or s.untyped_storage().data_ptr() == d.untyped_storage().data_ptr()):
            records[i] = None
    if len(records) > 8 or None in records or any(d.device != dev for _, d in pairs):
        for s, d in pairs:
            d.copy_(s)
        return
    arr = (_lib.RowCopy * len(records))(*records)
    with on_device(dev):
        rc = _lib.lib().adacode_copy_rows(ctypes.addressof(arr), len(records), stream_ptr(dev))
    _lib.check(rc, 'adacode_copy_rows')
    increment_version([d for _, d in pairs])
