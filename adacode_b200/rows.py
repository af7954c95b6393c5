"""Copies of dense token rows (a token's keys and values appended to the residual, the not yet packed tails behind the
segments) and what every launch needs of the device: its current stream, its being the current one."""
from __future__ import annotations

import contextlib
import ctypes
from typing import Optional, Sequence

import torch

from . import _lib

_HERE = contextlib.nullcontext()


def stream_ptr(device: torch.device) -> int:
    """Handle of the device's current stream."""
    index = device.index
    return torch._C._cuda_getCurrentRawStream(torch.cuda.current_device() if index is None else index)


def on_device(device: torch.device):
    """``torch.cuda.device(device)``, which costs as much as a launch, only where another device is current."""
    index = device.index
    return _HERE if index is None or index == torch.cuda.current_device() else torch.cuda.device(device)


def row_record(src: torch.Tensor, dst: torch.Tensor) -> Optional[tuple]:
    """``dst.copy_(src)`` as a record of the row-copy kernel, or None if it is not one: it takes plain bf16 CUDA tensors
    of one [B, H, T, D] shape on one device, rows on 16-byte boundaries, and no gradient to record."""
    if type(src) is not torch.Tensor or type(dst) is not torch.Tensor:
        return None
    if src.dtype != torch.bfloat16 or dst.dtype != torch.bfloat16 or not src.is_cuda or src.device != dst.device:
        return None
    shape = src.shape
    if len(shape) != 4 or shape != dst.shape or ((src.requires_grad or dst.requires_grad) and torch.is_grad_enabled()):
        return None
    a, b, c, u = src.stride()
    d, e, f, v = dst.stride()
    from_ptr, to_ptr = src.data_ptr(), dst.data_ptr()
    B, H, T, D = shape
    if u != 1 or v != 1 or (a | b | c | d | e | f | D) & 7 or (from_ptr | to_ptr) & 15 or B * H * T * D >= 2 ** 31:
        return None
    return (from_ptr, to_ptr, a, b, c, d, e, f, B, H, T, D)


def copy_rows(pairs: Sequence[tuple]) -> None:
    """``dst.copy_(src)`` for every ``(src, dst)`` pair, in one launch where the kernel takes all of them.

    The caches do not use it: describing two one-token tensors costs more on the host than the launch it saves
    (keys and values of a token appended: 21.5 us, two ``copy_`` calls 19.5 us)."""
    pairs = [(s, d) for s, d in pairs if d.numel()]
    if not pairs:
        return
    dev = pairs[0][1].device
    records = [row_record(s, d) for s, d in pairs]
    if len(records) > 8 or None in records or any(d.device != dev for _, d in pairs):
        for s, d in pairs:
            d.copy_(s)
        return
    arr = (_lib.RowCopy * len(records))(*records)
    with on_device(dev):
        rc = _lib.lib().adacode_copy_rows(ctypes.addressof(arr), len(records), stream_ptr(dev))
    _lib.check(rc, 'adacode_copy_rows')
