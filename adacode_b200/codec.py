"""Tiled float11 codec: torch-facing wrappers over the sm_100a kernels.

Mirrors the interface of the reference's ``compress_tiled_kv.py`` (``compress_tiled_tensor``,
``TiledCompressedTensor``, ``materialize_tiled_state``) and adds the batched forms the cache
uses: one launch packs every 128-token block of a prefill (``pack_blocks``), one launch
unpacks any list of segments (``unpack_segments``).

All tensors are CUDA tensors; kernels run on ``torch.cuda.current_stream``.  There is no CPU
path: on a CPU tensor, or without the built library, these functions raise.
"""
from __future__ import annotations

import ctypes
import threading
from dataclasses import dataclass, field
from typing import Any, Optional, Sequence

import torch

from . import _lib
from .rows import increment_version, on_device, row_record, stream_ptr

_SUPPORTED_TILE_NBITS = (1, 2, 3, 4)
_DEFAULT_TILE_NBITS = 3


# --------------------------------------------------------------------------------------
# per-device scratch
# --------------------------------------------------------------------------------------

# Streams of a GPU that keep buffers; beyond it the oldest one's go back to the allocator.
_MAX_STREAMS = 8


class _StreamBuffers:
    """Memory that launches hand data on in: one buffer per stream of a GPU (two streams are not ordered), grown on demand."""

    def __init__(self, device: torch.device, make):
        self.device, self.make = device, make
        self.by_stream: dict[int, torch.Tensor] = {}      # oldest first
        self.lock = threading.Lock()

    def get(self, stream: int, need: int) -> torch.Tensor:
        """At least ``need`` bytes for ``stream``, the current one: they are allocated on it, so a buffer that was replaced
        or dropped is used again in the stream's order."""
        buf = self.by_stream.get(stream)
        if buf is None or buf.numel() < need:
            buf = self.make(max(1 << 20, need + need // 4 + 256), dtype=torch.uint8, device=self.device)
            with self.lock:
                self.by_stream.pop(stream, None)
                self.by_stream[stream] = buf
                while len(self.by_stream) > _MAX_STREAMS:
                    del self.by_stream[next(iter(self.by_stream))]
        return buf


class _DeviceScratch:
    """The pack scratch, the memory for the fused attention's partial results and the status word of one GPU."""

    def __init__(self, device: torch.device):
        self.device = device
        self.packs = _StreamBuffers(device, torch.zeros)  # (the library wants a zero-filled scratch and leaves it reusable)
        self.partials = _StreamBuffers(device, torch.empty)
        self.status = torch.zeros(2, dtype=torch.int32, device=device)

    def workspace_for(self, n_tiles: int, tile_elems: int) -> torch.Tensor:
        """The current stream's pack scratch."""
        return self.packs.get(stream_ptr(self.device), int(_lib.lib().adacode_pack_workspace_bytes(n_tiles, tile_elems)))


_scratch: dict[torch.device, _DeviceScratch] = {}


def _scratch_for(device: torch.device) -> _DeviceScratch:
    s = _scratch.get(device)
    if s is not None:
        return s
    device = torch.device(device)
    if device.type != 'cuda':
        raise _lib.AdacodeError(f'float11 kernels need a CUDA tensor, got device {device} (there is no CPU path)')
    if device.index is None:
        device = torch.device('cuda', torch.cuda.current_device())
    s = _scratch.get(device)
    if s is None:
        s = _scratch[device] = _DeviceScratch(device)
    return s


class _Mailbox(threading.local):
    """A thread's page-locked host bytes that ``read_back``'s kernel writes into."""

    def __init__(self):
        self.bytes: Optional[torch.Tensor] = None
        self.events: dict[torch.device, torch.cuda.Event] = {}


_mailbox = _Mailbox()


def read_back(t: torch.Tensor):
    """Host copy (numpy array of ``t``'s shape and dtype) of a small device tensor.

    The reference reads such values with ``.to('cpu')`` / ``.item()`` (escape totals,
    compress_tiled_kv.py:559-588; histograms, float_cache_utils.py:373), i.e. with cudaMemcpy, which
    queues behind whatever bulk transfer occupies the copy engine.  Here a one-CTA kernel stores the
    bytes into pinned host memory (``adacode_copy_to_host``) and the host waits for an event."""
    if not t.is_contiguous():
        t = t.contiguous()
    nbytes = t.numel() * t.element_size()
    if nbytes == 0 or nbytes % 4 != 0 or nbytes > (1 << 20):
        return t.cpu().numpy()
    dev = t.device
    _scratch_for(dev)
    box = _mailbox
    if box.bytes is None or box.bytes.numel() < nbytes:
        box.bytes = torch.empty(max(1 << 16, nbytes), dtype=torch.uint8).pin_memory()
    event = box.events.get(dev)
    if event is None:
        event = box.events[dev] = torch.cuda.Event()
    stream = torch.cuda.current_stream(dev)
    with on_device(dev):
        rc = _lib.lib().adacode_copy_to_host(t.data_ptr(), box.bytes.data_ptr(), nbytes, int(stream.cuda_stream))
    if rc == _lib.ERR_INVALID_ARG:
        return t.cpu().numpy()           # pinned memory this device cannot address: plain copy
    _lib.check(rc, 'adacode_copy_to_host')
    event.record(stream)
    event.synchronize()
    import numpy as np
    out = box.bytes[:nbytes].numpy().copy()
    return out.view(np.dtype(str(t.dtype).replace('torch.', ''))).reshape(tuple(t.shape))


def check_device_status(device) -> None:
    """Read the device status word (synchronises) and raise if a kernel flagged a problem."""
    s = _scratch_for(torch.device(device))
    word = int(read_back(s.status)[0])
    if word:
        s.status.zero_()
        raise _lib.AdacodeError('device status: ' + describe_status(word))


_STATUS_TEXT = (
    (_lib.STATUS_ESCAPE_OVERFLOW, 'escape buffer too small during pack'),
    (_lib.STATUS_ESCAPE_UNDERRUN, 'escape list shorter than the code plane requires during unpack'),
    (_lib.STATUS_TIMEOUT, 'a bounded on-chip wait gave up (results of that launch are invalid)'),
    (_lib.STATUS_MISALIGNED, 'a plane pointer in a segment record is not 16-byte aligned (tile skipped)'),
)


def describe_status(word: int) -> str:
    """Text for the bits of a device status word (every bit is named; unknown bits are shown in hex)."""
    parts = [text for bit, text in _STATUS_TEXT if word & bit]
    rest = word & ~sum(bit for bit, _ in _STATUS_TEXT)
    if rest:
        parts.append(f'unknown status bits {rest:#x}')
    return '; '.join(parts) if parts else 'ok'


# --------------------------------------------------------------------------------------
# containers
# --------------------------------------------------------------------------------------

@dataclass
class TiledCompressedTensor:
    """One packed block, field for field the reference's dataclass
    (compress_tiled_kv.py:238-342)."""

    sign_mass_data: torch.Tensor
    exp_data: torch.Tensor
    invalid_exp: torch.Tensor
    tile_invalid_base: torch.Tensor
    left: int
    right: int
    nbits: int
    original_shape: tuple
    seq_tile_size: int
    head_dim: int
    tile_head_dim: int
    tile_num_lanes: int
    num_sequence_tiles: int
    num_kv_heads: int
    device: torch.device
    layout: str = 'tiled'
    decode_kind: str = 'tiled_decode'
    has_outliers: bool = True

    @property
    def n_elements(self) -> int:
        n = 1 if self.original_shape else 0
        for d in self.original_shape:
            n *= d
        return n

    def get_memory(self) -> dict:
        """compress_tiled_kv.py:269-282."""
        compressed = (self.sign_mass_data.numel() + self.exp_data.numel() + self.invalid_exp.numel()
                      + self.tile_invalid_base.numel() * self.tile_invalid_base.element_size())
        original = self.n_elements * 2
        return {
            'compressed_memory': compressed,
            'original_memory': original,
            'ratio': 0.0 if original == 0 else compressed / original,
        }

    def export_state(self) -> dict:
        """compress_tiled_kv.py:284-306."""
        state = {
            'layout': self.layout, 'right': self.right, 'nbits': self.nbits, 'left': self.left,
            'device': self.device, 'original_shape': self.original_shape,
            'sign_mass_data': self.sign_mass_data, 'exp_data': self.exp_data,
            'seq_tile_size': self.seq_tile_size, 'head_dim': self.head_dim,
            'tile_head_dim': self.tile_head_dim, 'tile_num_lanes': self.tile_num_lanes,
            'num_sequence_tiles': self.num_sequence_tiles, 'num_kv_heads': self.num_kv_heads,
            'n_elements': self.n_elements, 'has_outliers': self.has_outliers,
        }
        if self.has_outliers:
            state['invalid_exp'] = self.invalid_exp
            state['tile_invalid_base'] = self.tile_invalid_base
        return state

    def export_decode_view(self) -> dict:
        state = self.export_state()
        state['kind'] = self.decode_kind
        return state

    def materialize(self) -> torch.Tensor:
        """compress_tiled_kv.py:313-337."""
        B, H, S, D = self.original_shape
        out = torch.empty((B, H, S, D), dtype=torch.bfloat16, device=self.sign_mass_data.device)
        unpack_segments([self], out)
        return out


class SegmentRef:
    """Handle on segment ``j`` of a ``PackedChunk``: everything the cache's bookkeeping needs
    (window, shape, escape count, byte accounting) is arithmetic on the chunk, so a prefill of
    hundreds of blocks creates no per-block tensor views; ``view()`` materialises the reference-
    shaped ``TiledCompressedTensor`` on demand."""

    __slots__ = ('chunk', 'j')

    def __init__(self, chunk: 'PackedChunk', j: int):
        self.chunk = chunk
        self.j = int(j)

    left = property(lambda self: self.chunk.left)
    right = property(lambda self: self.chunk.right)
    nbits = property(lambda self: self.chunk.nbits)
    seq_tile_size = property(lambda self: self.chunk.seq_tile)
    head_dim = property(lambda self: self.chunk.head_dim)

    @property
    def original_shape(self) -> tuple:
        c = self.chunk
        return (c.batch, c.heads, c.seq_tile, c.head_dim)

    @property
    def n_elements(self) -> int:
        c = self.chunk
        return c.batch * c.heads * c.seq_tile * c.head_dim

    @property
    def n_escapes(self) -> int:
        off = self.chunk.seg_offsets
        return int(off[self.j + 1]) - int(off[self.j])

    def view(self) -> TiledCompressedTensor:
        return self.chunk.segment(self.j)

    # tensor fields, for code written against TiledCompressedTensor
    sign_mass_data = property(lambda self: self.view().sign_mass_data)
    exp_data = property(lambda self: self.view().exp_data)
    invalid_exp = property(lambda self: self.view().invalid_exp)
    tile_invalid_base = property(lambda self: self.view().tile_invalid_base)

    def get_memory(self) -> dict:
        """compress_tiled_kv.py:269-282, without touching a tensor."""
        c = self.chunk
        n = self.n_elements
        compressed = n + n * c.nbits // 8 + self.n_escapes + 4 * c.batch * c.heads
        return {'compressed_memory': compressed, 'original_memory': 2 * n,
                'ratio': 0.0 if n == 0 else compressed / (2 * n)}

    def export_state(self) -> dict:
        return self.view().export_state()

    def export_decode_view(self) -> dict:
        return self.view().export_decode_view()

    def materialize(self) -> torch.Tensor:
        return self.view().materialize()


@dataclass
class PackedChunk:
    """``n_blocks`` consecutive segments produced by one pack launch with one window.
    Plane tensors are segment-major; ``segment(j)`` gives views shaped like the reference's
    per-block ``TiledCompressedTensor``."""

    sign_mant: torch.Tensor      # uint8 [n_blocks, B*H*tile_elems]
    codes: torch.Tensor          # uint8 [n_blocks, B*H*tile_elems*nbits/8]
    escapes: torch.Tensor        # uint8 [n_escapes]
    tile_base: torch.Tensor      # int32 [n_blocks, B*H]
    seg_offsets: list            # host ints, n_blocks + 1
    seg_offsets_dev: torch.Tensor  # the same, int64 on the device
    left: int
    right: int
    nbits: int
    batch: int
    heads: int
    seq_tile: int
    head_dim: int
    _segments: dict = field(default_factory=dict, repr=False)

    @property
    def n_blocks(self) -> int:
        return int(self.sign_mant.shape[0])

    @property
    def n_escapes(self) -> int:
        return int(self.seg_offsets[-1])

    def segment(self, j: int) -> TiledCompressedTensor:
        seg = self._segments.get(j)
        if seg is None:
            lo, hi = int(self.seg_offsets[j]), int(self.seg_offsets[j + 1])
            seg = TiledCompressedTensor(
                sign_mass_data=self.sign_mant[j], exp_data=self.codes[j], invalid_exp=self.escapes[lo:hi],
                tile_invalid_base=self.tile_base[j], left=self.left, right=self.right, nbits=self.nbits,
                original_shape=(self.batch, self.heads, self.seq_tile, self.head_dim),
                seq_tile_size=self.seq_tile, head_dim=self.head_dim, tile_head_dim=self.head_dim,
                tile_num_lanes=self.head_dim // 8, num_sequence_tiles=1, num_kv_heads=self.heads,
                device=self.sign_mant.device)
            self._segments[j] = seg
        return seg

    def segments(self) -> list:
        """Cheap handles, one per block (``SegmentRef``)."""
        return [SegmentRef(self, j) for j in range(self.n_blocks)]


# --------------------------------------------------------------------------------------
# kernels
# --------------------------------------------------------------------------------------

def _check_src(x: torch.Tensor) -> torch.Tensor:
    if x.dtype != torch.bfloat16:
        x = x.to(torch.bfloat16)
    if x.dim() != 4:
        raise ValueError(f'Expected 4D [batch, kv_heads, seq, head_dim] tensor, got {tuple(x.shape)}')
    if x.shape[-1] % 8 != 0:
        raise ValueError(f'Tiled compressed path requires head_dim % 8 == 0, got {x.shape[-1]}')
    sb, sh, ss, sd = x.stride()
    if x.numel() and (sd != 1 or (sb | sh | ss) % 8 != 0 or x.data_ptr() % 16 != 0):
        x = x.contiguous()
    return x


class _PendingPack:
    """One tensor of a pack: what was asked for, and the outputs of its launch."""

    def __init__(self, **kw):
        self.__dict__.update(kw)


def _check_blocks(S: int, seq_tile: int) -> None:
    if seq_tile <= 0:
        raise ValueError('seq_tile_size must be positive')
    if S % seq_tile != 0:
        raise ValueError(f'sequence length {S} is not a multiple of seq_tile_size {seq_tile}')


def _default_escape_capacity(n: int, nbits: int) -> int:
    """Room for an eighth of the elements, more for the windows of one and of three exponents, of which a third to a
    half of the elements fall outside: a buffer that is too small costs a second pack of the whole span."""
    share = n // 8 if nbits > 2 else n // 2 if nbits == 2 else n
    return min(max(4096, share), max(n, 1))


def _pack_again(p: _PendingPack, capacity: int) -> torch.Tensor:
    """Pack ``p`` into its planes once more, with room for ``capacity`` escapes; its histogram is complete."""
    ws = _scratch_for(p.dev).workspace_for(p.B * p.H * p.n_blocks, p.seq_tile * p.D)
    esc = torch.empty(capacity, dtype=torch.uint8, device=p.dev)
    sb, sh, ss, _ = p.x.stride()
    with on_device(p.dev):
        rc = _lib.lib().adacode_pack_tiles(
            p.x.data_ptr(), sb, sh, ss, p.B, p.H, p.n_blocks, p.seq_tile, p.D, p.right, p.nbits,
            p.sign_mant.data_ptr(), p.codes.data_ptr(), esc.data_ptr(), capacity, p.tile_base.data_ptr(),
            p.meta.data_ptr(), 0, ws.data_ptr(), ws.numel(), p.meta.data_ptr() + 8 * (p.n_blocks + 1), stream_ptr(p.dev))
    _lib.check(rc, 'adacode_pack_tiles')
    return esc


def _pack_now(xs: Sequence[torch.Tensor], rights: Sequence[int], nbits: Sequence[int], seq_tile: int, need_hist, capacities: Sequence):
    """Pack tensors (in one launch those that share shape and code length, as the keys and the values of a span do),
    wait for the escape totals and finish.  ``need_hist``: whether, or for a single tensor the int32[256] device histogram
    to add to.
    Returns ``[(PackedChunk, device histogram or None), ...]`` and the new histograms on the host (int32 [n, 256]) or None."""
    pending, caps, tiles, tile_elems = [], [], 0, 0
    for x, right, bits, cap in zip(xs, rights, nbits, capacities):
        if bits not in _SUPPORTED_TILE_NBITS:
            raise ValueError(f'Tiled compressed path supports nbits in {_SUPPORTED_TILE_NBITS}, got {bits}')
        x = _check_src(x)
        B, H, S, D = x.shape
        _check_blocks(S, seq_tile)
        n, n_blocks = B * H * S * D, S // seq_tile
        guessed = cap is None
        cap = _default_escape_capacity(n, bits) if guessed else min(int(cap), max(n, 1))
        pending.append(_PendingPack(x=x, right=right, nbits=bits, seq_tile=seq_tile, B=B, H=H, D=D, n_blocks=n_blocks, dev=x.device,
                                    n=n, guessed=guessed, cap=cap))
        caps.append(cap)
        tiles, tile_elems = tiles + B * H * n_blocks, max(tile_elems, seq_tile * D)
    ws = _scratch_for(pending[0].dev).workspace_for(tiles, tile_elems)
    parts, host_hist = _lib.native().pack(tuple([p.x for p in pending]), tuple(rights), tuple(nbits), seq_tile, tuple(caps), need_hist, ws)
    out = []
    for p, part in zip(pending, parts):
        p.sign_mant, p.codes, p.escapes, p.tile_base, p.meta, p.hist, offsets, status = part
        out.append(_finish_pack(p, offsets, status))
    if host_hist is not None:
        import numpy as np
        host_hist = np.frombuffer(host_hist, dtype=np.int32).reshape(len(xs), 256).copy()
    return out, host_hist


def _trim_escapes(escapes: torch.Tensor, total: int, large_guess: bool, n: int) -> torch.Tensor:
    # (a large first guess is not kept, which packs of single blocks would for the cache's life: it is cut to size
    # where an eighth more than the escapes and a 32nd of the elements are unused)
    keep = total + total // 8 + min(65536, n // 32) if large_guess else 2 * total + 65536
    return escapes[:total].clone() if escapes.numel() > keep else escapes[:total]


def _finish_pack(p: _PendingPack, offsets: list, status: int):
    n_blocks = p.n_blocks
    total = offsets[-1]
    escapes = p.escapes
    # the kernels flag an overflow exactly when a stream does not fit its buffer; packs that shared
    # a launch share the status word, so each one decides by its own total
    status_other = status & ~_lib.STATUS_ESCAPE_OVERFLOW
    if total > p.cap:
        p.meta = torch.zeros(n_blocks + 2, dtype=torch.int64, device=p.dev)
        escapes = _pack_again(p, total)
        host = read_back(p.meta)
        if int(host[n_blocks + 1]) & 0xFFFFFFFF:
            raise _lib.AdacodeError('adacode_pack_tiles: escape overflow after re-run with exact capacity')
    elif status_other:
        raise _lib.AdacodeError(f'adacode_pack_tiles: device status {status:#x} ({describe_status(status)})')
    escapes = _trim_escapes(escapes, total, p.guessed and p.nbits <= 2, p.n)
    meta = p.meta if p.meta.shape[0] == n_blocks + 1 else p.meta[: n_blocks + 1]
    chunk = PackedChunk(p.sign_mant, p.codes, escapes, p.tile_base, offsets, meta,
                        p.right - 2 ** p.nbits + 1, p.right, p.nbits, p.B, p.H, p.seq_tile, p.D)
    return chunk, p.hist


def pack_blocks(x: torch.Tensor, right: int, nbits: int, seq_tile: int = 128, need_hist: bool = False,
                hist_out: Optional[torch.Tensor] = None, escape_capacity: Optional[int] = None):
    """Pack ``x`` [B, H, n_blocks*seq_tile, D] (bf16, any B/H/S strides) into ``n_blocks`` segments
    with the window ``(right - 2**nbits + 1, right]`` in one launch.

    Returns ``(PackedChunk, hist)``; ``hist`` is an int32[256] device tensor of all exponents when
    ``need_hist`` (``hist_out`` is added to instead when given).  One small device-to-host read
    (segment escape totals and the status word) ends the call.
    """
    [done], _ = _pack_now([x], [int(right)], [int(nbits)], seq_tile, hist_out if need_hist and hist_out is not None else need_hist,
                          [escape_capacity])
    return done


def pack_pair(k: torch.Tensor, v: torch.Tensor, k_params, v_params, seq_tile: int = 128, need_hist: bool = False,
              capacities=(None, None)):
    """Pack the keys and the values of one span, with one launch and one round trip to the host where they have one
    shape and code length: segment offsets, status and (with ``need_hist``) exponent histograms come back together.  Returns
    ``(k_chunk, v_chunk, k_hist, v_hist, k_hist_host, v_hist_host)``; the ``*_host`` entries are
    numpy int32[256] copies of the histograms (None without ``need_hist``)."""
    # (keys and values of one shape and code length go through ONE launch, their windows may differ)
    (kd, vd), hists = _pack_now([k, v], [int(k_params[0]), int(v_params[0])], [int(k_params[1]), int(v_params[1])], seq_tile,
                                need_hist, capacities)
    kh, vh = (None, None) if hists is None else hists
    return kd[0], vd[0], kd[1], vd[1], kh, vh


def pack_flat(x: torch.Tensor, right: int, nbits: int, block_elems: int, hist: Optional[torch.Tensor] = None) -> tuple:
    """``(sign_mant, codes, escapes, block_base int32)`` of a contiguous bf16 CUDA tensor in the flat layout, whose
    element count is a multiple of 8; ``hist`` (int32[256] on the device) is added to."""
    n = x.numel()
    if x.data_ptr() % 16:
        x = x.clone()                            # (a view may begin anywhere, the kernels want 16-byte boundaries)
    dev = x.device
    cap, guessed = _default_escape_capacity(n, nbits), True
    while True:
        ws = _scratch_for(dev).workspace_for(n // block_elems, block_elems)
        sm, cd, escapes, base, total, status = _lib.native().pack_flat(x, right, nbits, block_elems, cap, hist if guessed else None, ws)
        if total <= cap:
            break
        if not guessed:
            raise _lib.AdacodeError('adacode_pack_flat: escape overflow after re-run with exact capacity')
        cap, guessed = total, False              # (the histogram is complete from the first pass)
    if status:
        raise _lib.AdacodeError(f'adacode_pack_flat: device status {status:#x} ({describe_status(status)})')
    return sm, cd, _trim_escapes(escapes, total, guessed and nbits <= 2, n), base


def unpack_chunk(chunk: PackedChunk, dst: torch.Tensor, seq_offset: int = 0) -> None:
    """Unpack every segment of ``chunk`` into ``dst[:, :, seq_offset : seq_offset + n_blocks*seq_tile]``."""
    B, H, T, D = chunk.batch, chunk.heads, chunk.seq_tile, chunk.head_dim
    _check_dst(dst, B, H, D, seq_offset + chunk.n_blocks * T)
    dev = dst.device
    sc = _scratch_for(dev)
    view = dst[:, :, seq_offset:]
    db, dh, ds, _ = dst.stride()
    seg_off = chunk.seg_offsets_dev
    with on_device(dev):
        rc = _lib.lib().adacode_unpack_tiles(
            chunk.sign_mant.data_ptr(), chunk.codes.data_ptr(), chunk.escapes.data_ptr(), chunk.escapes.numel(),
            chunk.tile_base.data_ptr(), seg_off.data_ptr(), B, H, chunk.n_blocks, T, D,
            chunk.left, chunk.nbits, view.data_ptr(), db, dh, ds, sc.status.data_ptr(), stream_ptr(dev))
    _lib.check(rc, 'adacode_unpack_tiles')


def _check_dst(dst: torch.Tensor, B: int, H: int, D: int, min_seq: int) -> None:
    shape = dst.shape
    if dst.dtype != torch.bfloat16 or len(shape) != 4:
        raise ValueError(f'dst must be a 4D bf16 tensor, got {dst.dtype} {tuple(dst.shape)}')
    B2, H2, S2, D2 = shape
    if B2 != B or H2 != H or D2 != D or S2 < min_seq:
        raise ValueError(f'dst shape {tuple(dst.shape)} cannot hold [{B}, {H}, {min_seq}, {D}]')
    if dst.stride(3) != 1:
        raise ValueError('dst must have unit stride along head_dim')


_SEGMENT_DTYPE = None


def _segment_dtype():
    """numpy mirror of ``struct adacode_segment`` (56 bytes)."""
    global _SEGMENT_DTYPE
    if _SEGMENT_DTYPE is None:
        import numpy as np
        _SEGMENT_DTYPE = np.dtype([('sign_mant', '<u8'), ('codes', '<u8'), ('escapes', '<u8'), ('tile_base', '<u8'),
                                   ('escapes_len', '<i8'), ('dst_seq_offset', '<i8'), ('left', '<i4'),
                                   ('nbits', '<i4')])
        assert _SEGMENT_DTYPE.itemsize == ctypes.sizeof(_lib.Segment)
    return _SEGMENT_DTYPE


def _check_segment_buffers(seg) -> None:
    """A segment record carries raw pointers: refuse on the host what would fault on the device."""
    B, H, T, D = (int(v) for v in seg.original_shape)
    n = B * H * T * D
    nbits = int(seg.nbits)
    if nbits not in _SUPPORTED_TILE_NBITS:
        raise ValueError(f'Tiled compressed path supports nbits in {_SUPPORTED_TILE_NBITS}, got {nbits}')
    if seg.sign_mass_data.dtype != torch.uint8 or seg.sign_mass_data.numel() < n:
        raise ValueError(f'segment sign_mass_data must hold {n} uint8 values, got {seg.sign_mass_data.numel()}')
    if seg.exp_data.dtype != torch.uint8 or seg.exp_data.numel() < n * nbits // 8:
        raise ValueError(f'segment exp_data must hold {n * nbits // 8} uint8 values, got {seg.exp_data.numel()}')
    base = seg.tile_invalid_base
    if base.dtype != torch.int32 or base.numel() < B * H or not base.is_contiguous():
        raise ValueError(f'segment tile_invalid_base must be {B * H} contiguous int32 values, got '
                         f'{base.numel()} of {base.dtype}')
    if n and (seg.sign_mass_data.data_ptr() % 16 or seg.exp_data.data_ptr() % 16):
        raise ValueError('segment planes must start on 16-byte boundaries')
    if seg.invalid_exp.numel() and seg.invalid_exp.dtype != torch.uint8:
        raise ValueError('segment invalid_exp must be uint8')


def build_segment_table(segments: Sequence, seq_offsets: Optional[Sequence[int]] = None,
                        device=None) -> torch.Tensor:
    """Device array of ``adacode_segment`` records (as uint8) for ``unpack_segments``.
    ``seq_offsets[i]`` is segment i's first token in the destination; the default stacks the
    segments one after the other.  Runs of ``SegmentRef`` from one chunk are filled with array
    arithmetic on the chunk's base pointers, so a table over hundreds of blocks costs a handful
    of numpy operations."""
    import numpy as np
    n = len(segments)
    table = np.zeros(max(n, 1), dtype=_segment_dtype())
    i = 0
    run_tokens = 0
    while i < n:
        seg = segments[i]
        if isinstance(seg, SegmentRef):
            c = seg.chunk
            k = i + 1
            while k < n and isinstance(segments[k], SegmentRef) and segments[k].chunk is c \
                    and segments[k].j == segments[k - 1].j + 1:
                k += 1
            js = np.arange(seg.j, seg.j + (k - i), dtype=np.int64)
            offs = np.asarray(c.seg_offsets, dtype=np.int64)
            bh = c.batch * c.heads
            tile = c.seq_tile * c.head_dim
            rows = table[i:k]
            rows['sign_mant'] = c.sign_mant.data_ptr() + js * (bh * tile)
            rows['codes'] = c.codes.data_ptr() + js * (bh * tile * c.nbits // 8)
            esc_base = c.escapes.data_ptr() if c.escapes.numel() else 0
            lens = offs[js + 1] - offs[js]
            rows['escapes'] = np.where(lens > 0, esc_base + offs[js], 0)
            rows['tile_base'] = c.tile_base.data_ptr() + js * (4 * bh)
            rows['escapes_len'] = lens
            rows['left'] = c.left
            rows['nbits'] = c.nbits
            tokens = np.full(k - i, c.seq_tile, dtype=np.int64)
        else:
            k = i + 1
            rows = table[i:k]
            _check_segment_buffers(seg)
            rows['sign_mant'] = seg.sign_mass_data.data_ptr()
            rows['codes'] = seg.exp_data.data_ptr()
            rows['escapes'] = seg.invalid_exp.data_ptr() if seg.invalid_exp.numel() else 0
            rows['tile_base'] = seg.tile_invalid_base.data_ptr()
            rows['escapes_len'] = seg.invalid_exp.numel()
            rows['left'] = int(seg.left)
            rows['nbits'] = int(seg.nbits)
            tokens = np.asarray([int(seg.original_shape[-2])], dtype=np.int64)
        if seq_offsets is None:
            starts = run_tokens + np.concatenate(([0], np.cumsum(tokens)[:-1]))
            run_tokens += int(tokens.sum())
        else:
            starts = np.asarray([int(v) for v in seq_offsets[i:k]], dtype=np.int64)
            run_tokens = int(starts[-1] + tokens[-1])
        rows['dst_seq_offset'] = starts
        i = k
    host = torch.from_numpy(table[:n].view(np.uint8).reshape(-1).copy()) if n else torch.empty(0, dtype=torch.uint8)
    if device is None:
        s0 = segments[0]
        device = s0.chunk.sign_mant.device if isinstance(s0, SegmentRef) else s0.sign_mass_data.device
    return host.to(device, non_blocking=False)


def unpack_segments(segments: Sequence[TiledCompressedTensor], dst: torch.Tensor,
                    seq_offsets: Optional[Sequence[int]] = None, table: Optional[torch.Tensor] = None) -> None:
    """Unpack a list of segments (any mix of windows and code lengths) into ``dst`` [B, H, S, D]
    with one launch.  Replaces the reference's per-segment decode + ``torch.cat``
    (float_cache_utils.py:1257-1264)."""
    if not segments:
        return
    first = segments[0]
    B, H, T, D = first.original_shape
    _check_one_shape(segments, (B, H, T, D))
    _check_dst(dst, B, H, D, 0)
    dev = dst.device
    sc = _scratch_for(dev)
    if table is None:
        table = build_segment_table(segments, seq_offsets, dev)
    db, dh, ds, _ = dst.stride()
    with on_device(dev):
        rc = _lib.lib().adacode_unpack_segments(table.data_ptr(), len(segments), B, H, T, D, dst.data_ptr(),
                                                db, dh, ds, sc.status.data_ptr(), stream_ptr(dev))
    _lib.check(rc, 'adacode_unpack_segments')


def device_status(device: torch.device) -> torch.Tensor:
    """The status word of a GPU that unpack launches write to."""
    return _scratch_for(device).status


def check_one_shape(segs: Sequence) -> None:
    """Refuse a list whose segments differ in [batch, kv_heads, seq_tile, head_dim]."""
    if segs:
        _check_one_shape(segs, tuple(segs[0].original_shape))


def _check_one_shape(segs: Sequence, shape0: tuple) -> None:
    """Refuse segments of another [batch, kv_heads, seq_tile, head_dim]; segments of one chunk have one shape."""
    try:
        chunk = segs[0].chunk                 # (of most segments: the prefill's)
        rest = [seg for seg in segs if seg.chunk is not chunk]
    except AttributeError:                    # others than SegmentRef among them
        chunk, rest = None, segs
    for seg in rest if chunk is None else (segs[0], *rest):
        if tuple(seg.original_shape) != shape0:
            raise ValueError('all segments of one call must share [batch, kv_heads, seq_tile, head_dim]')


def unpack_segments_multi(jobs: Sequence[tuple]) -> None:
    """Unpack several segment lists, each into its own destination, with ONE launch when they
    share [batch, kv_heads, seq_tile, head_dim] (the keys and the values of a layer).
    ``jobs``: ``(segments, dst, table_or_None)`` tuples; anything that does not fit one launch
    falls back to one ``unpack_segments`` call per entry."""
    jobs = [j for j in jobs if j[0]]
    if not jobs:
        return
    shape0 = tuple(jobs[0][0][0].original_shape)
    same = all(tuple(seg.original_shape) == shape0 for segs, _, _ in jobs for seg in (segs[0], segs[-1]))
    if len(jobs) == 1 or not same or len(jobs) > int(_lib.lib().adacode_max_jobs()):
        for segs, dst, table in jobs:
            unpack_segments(segs, dst, table=table)
        return
    _unpack_with_rows([(segs, dst, table, None) for segs, dst, table in jobs], shape0)


def _unpack_with_rows(jobs: Sequence[tuple], shape: tuple) -> None:
    B, H, T, D = shape
    dev = jobs[0][1].device
    records, rows, keep = [], [], []
    for segs, dst, table, row in jobs:
        _check_one_shape(segs, shape)
        _check_dst(dst, B, H, D, 0)
        if table is None:
            table = build_segment_table(segs, None, dev)
        keep.append(table)
        db, dh, ds, _ = dst.stride()
        records.append((table.data_ptr(), len(segs), 0, dst.data_ptr(), db, dh, ds))
        if row is not None:
            rows.append(row)
    arr = (_lib.UnpackJob * len(records))(*records)
    row_arr = (_lib.RowCopy * len(rows))(*rows) if rows else None
    with on_device(dev):
        rc = _lib.lib().adacode_unpack_jobs_with_rows(
            ctypes.addressof(arr), len(records), B, H, T, D, None if row_arr is None else ctypes.addressof(row_arr),
            len(rows), _scratch_for(dev).status.data_ptr(), stream_ptr(dev))
    _lib.check(rc, 'adacode_unpack_jobs_with_rows')


def unpack_with_tails(parts: Sequence[tuple], prefix: int, rows: int) -> None:
    """Dense keys and values of one layer: for every ``(segments, table, dense, tail)`` the segments are unpacked into
    the front of the contiguous ``dense`` [B, H, prefix + rows, D] and the first ``rows`` tokens of ``tail``
    [B, H, capacity, D] copied behind them, in one launch for parts of one shape.  A tail that is more than plain
    rows (see ``row_record``) is left to ``Tensor.copy_``."""
    jobs, shapes, left = [], [], []
    for segs, table, dense, tail in parts:
        shapes.append(tuple(segs[0].original_shape))
        if len(segs) * shapes[-1][2] > prefix or dense.shape[2] < prefix + rows:
            raise ValueError(f'{len(segs)} segments of {shapes[-1][2]} tokens and {rows} rows behind {prefix} '
                             f'do not fit {tuple(dense.shape)}')
        row = row_record(tail, dense, rows, prefix) if rows else None
        if rows and row is None:
            left.append((dense, tail))
        jobs.append((segs, dense, table, row))
    if all(s == shapes[0] for s in shapes):
        _unpack_with_rows(jobs, shapes[0])
    else:
        for job, shape in zip(jobs, shapes):
            _unpack_with_rows([job], shape)
    # (autograd has to know that memory that it may have saved was overwritten)
    increment_version([dense for _, dense, _, row in jobs if row is not None])
    for dense, tail in left:
        dense[:, :, prefix: prefix + rows].copy_(tail[:, :, :rows])


def exponent_hist(x: torch.Tensor, hist_out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """int32[256] device histogram of the exponent field of ``x`` [B, H, S, D]
    (float_cache_utils.py:883-891)."""
    x = _check_src(x)
    dev = x.device
    _scratch_for(dev)
    hist = hist_out if hist_out is not None else torch.empty(256, dtype=torch.int32, device=dev)
    B, H, S, D = x.shape
    sb, sh, ss, _ = x.stride()
    L = _lib.lib()
    with on_device(dev):
        rc = (L.adacode_hist_bf16 if hist_out is not None else L.adacode_hist_bf16_cleared)(
            x.data_ptr(), sb, sh, ss, B, H, S, D, hist.data_ptr(), stream_ptr(dev))
    _lib.check(rc, 'adacode_hist_bf16')
    return hist


def choose_params_device(hists: torch.Tensor) -> torch.Tensor:
    """(right, nbits) pairs, int32 [n, 2] on the device, for int32 histograms [n, 256];
    nbits == 0 marks a histogram for which no code length beats 8 bits."""
    if hists.dtype != torch.int32 or hists.shape[-1] != 256:
        raise ValueError('expected int32 histograms with 256 bins')
    h = hists.reshape(-1, 256).contiguous()
    dev = h.device
    _scratch_for(dev)
    out = torch.empty((h.shape[0], 2), dtype=torch.int32, device=dev)
    with on_device(dev):
        rc = _lib.lib().adacode_choose_params(h.data_ptr(), h.shape[0], out.data_ptr(), stream_ptr(dev))
    _lib.check(rc, 'adacode_choose_params')
    return out


def analysis_best_bits(data_freq, store_index: bool = False):
    """(right, nbits) for one 256-bin histogram given as a tensor, array or list on the host
    (float_cache_utils.py:373-398).  Raises IndexError where the reference does."""
    if store_index:
        raise NotImplementedError('store_index=True is not used by the float11 cache path')
    values = data_freq.tolist() if hasattr(data_freq, 'tolist') else list(data_freq)
    if len(values) != 256:
        raise ValueError(f'expected 256 bins, got {len(values)}')
    arr = (ctypes.c_int64 * 256)(*[int(v) for v in values])
    r, n = ctypes.c_int(0), ctypes.c_int(0)
    rc = _lib.lib().adacode_choose_params_host(arr, ctypes.byref(r), ctypes.byref(n))
    if rc == _lib.ERR_NO_CANDIDATE:
        raise IndexError('list index out of range')
    _lib.check(rc, 'adacode_choose_params_host')
    return int(r.value), int(n.value)


# --------------------------------------------------------------------------------------
# reference-shaped entry points
# --------------------------------------------------------------------------------------

def compress_tiled_tensor(original_data_bfloat16: torch.Tensor, right: int, nbits: int = _DEFAULT_TILE_NBITS,
                          seq_tile_size: int = 128, tile_head_dim: Optional[int] = None,
                          need_adjust: bool = False):
    """Pack exactly one block; same arguments, checks and return value as the reference
    (compress_tiled_kv.py:591-630)."""
    if nbits not in _SUPPORTED_TILE_NBITS:
        raise ValueError(f'Tiled compressed path supports nbits in {_SUPPORTED_TILE_NBITS}, got {nbits}')
    if original_data_bfloat16.dtype != torch.bfloat16:
        original_data_bfloat16 = original_data_bfloat16.to(torch.bfloat16)
    if original_data_bfloat16.dim() != 4:
        raise ValueError(
            f'Expected 4D [batch, kv_heads, seq, head_dim] tensor, got {tuple(original_data_bfloat16.shape)}')
    _, _, seq_len, head_dim = original_data_bfloat16.shape
    if seq_tile_size <= 0:
        raise ValueError('seq_tile_size must be positive')
    if tile_head_dim is None:
        tile_head_dim = head_dim
    if tile_head_dim != head_dim:
        raise ValueError(
            f'Tiled compressed path currently requires tile_head_dim == head_dim, got {tile_head_dim} vs {head_dim}')
    if head_dim % 8 != 0:
        raise ValueError(f'Tiled compressed path requires head_dim % 8 == 0, got {head_dim}')
    if seq_tile_size != seq_len:
        raise ValueError(
            'Tiled compressed path currently requires seq_tile_size == seq_len per compressed block, '
            f'got seq_tile_size={seq_tile_size}, seq_len={seq_len}')
    chunk, hist = pack_blocks(original_data_bfloat16, right, nbits, seq_tile_size, need_hist=need_adjust)
    return chunk.segment(0), hist


def tensor_from_state(state: dict) -> TiledCompressedTensor:
    dev = state['device']
    return TiledCompressedTensor(
        sign_mass_data=state['sign_mass_data'], exp_data=state['exp_data'],
        invalid_exp=state.get('invalid_exp', torch.empty((0,), dtype=torch.uint8, device=dev)),
        tile_invalid_base=state.get('tile_invalid_base', torch.empty((0,), dtype=torch.int32, device=dev)),
        left=state['left'], right=state['right'], nbits=state['nbits'],
        original_shape=tuple(state['original_shape']), seq_tile_size=state['seq_tile_size'],
        head_dim=state['head_dim'], tile_head_dim=state['tile_head_dim'],
        tile_num_lanes=state['tile_num_lanes'],
        num_sequence_tiles=int(state.get('num_sequence_tiles', 1)), num_kv_heads=state['num_kv_heads'],
        device=dev)


def materialize_tiled_state(state: dict) -> torch.Tensor:
    """Dense bf16 tensor of one exported segment state (compress_tiled_kv.py:754-791)."""
    if state.get('layout') == 'tiled_open_rows':
        raise NotImplementedError('open-row tiles are not produced by the segmented_tiled cache path')
    return tensor_from_state(state).materialize()
