"""Flat float11 codec: ``CompressorBitMap`` with the interface of the reference's
``compress_bitmap_merge.py`` (:633-873), served by the sm_100a kernels.

The flat layout packs ANY bf16 tensor (KV blocks of the 'legacy' cache layout, model weights) as
one sign/mantissa byte per element, n-bit exponent codes, one compact list of escaped exponents
in flat order and ``block_base``: the inclusive running escape count per ``invalid_block_size``
(= 128 x {8, 4, 8, 2}[nbits - 1]) elements.  ``compress`` is one ``adacode_pack_flat`` (for every 2**30
elements): tiles of one block each or, from 4 Mi elements on, of 16384 elements, and the end behind them
in one more launch; ``uncompress`` is one ``adacode_unpack_flat_ragged``, which decodes 16384-element
tiles, taking every (16384 / block)-th base, and the blocks behind them.  There is no CPU path.
"""
from __future__ import annotations

import torch

from . import _lib, codec
from .rows import on_device, stream_ptr

_BLOCK_GAPS = (8, 4, 8, 2)
_MAX_ELEMS_PER_CALL = 1 << 30


class CompressorBitMap:
    """reference: compress_bitmap_merge.py:633-873."""

    def __init__(self, right=129, nbits=3):
        self.device = None
        self.original_shape = None
        self.n_elements = None
        self.n_exp_data = None
        self.sign_mass_data = None
        self.exp_data = None
        self.invalid_exp = None
        self.blocksize = 128
        self.left = right - 2 ** nbits + 1
        self.right = right
        self.nbits = nbits
        self._configure_runtime()
        self.block_base = None          # int64, as the reference's torch.cumsum yields it
        self._base_i32 = None           # the same counts as the kernels read them

    def _configure_runtime(self):
        if self.nbits not in (1, 2, 3, 4):
            raise IndexError('list index out of range')          # the reference indexes a 4-entry list
        self.invalid_block_size = self.blocksize * _BLOCK_GAPS[self.nbits - 1]
        self.left_nbits = self.left << 7

    def reset_memory(self):
        self.device = None
        self.n_elements = None
        self.n_exp_data = None
        self.original_shape = None
        self.sign_mass_data = None
        self.exp_data = None
        self.invalid_exp = None
        self.block_base = None
        self._base_i32 = None

    def _update_compression_params(self, right, nbits):
        self.left = right - 2 ** nbits + 1
        self.right = right
        self.nbits = nbits
        self._configure_runtime()
        self.block_base = None

    def get_memory(self):
        if self.sign_mass_data is None:
            return {'compressed_memory': 0, 'original_memory': 0}
        compressed = (self.sign_mass_data.numel() + self.exp_data.numel()
                      + (0 if self.invalid_exp is None else self.invalid_exp.numel())
                      + (0 if self.block_base is None else self.block_base.numel() * self.block_base.element_size()))
        original = 0 if self.n_elements is None else self.n_elements * 2
        return {'compressed_memory': compressed, 'original_memory': original,
                'ratio': 0 if original == 0 else compressed / original}

    _STATE_KEYS = ('right', 'nbits', 'left', 'left_nbits', 'blocksize', 'invalid_block_size', 'device',
                   'original_shape', 'n_elements', 'n_exp_data', 'sign_mass_data', 'exp_data', 'invalid_exp',
                   'block_base')

    def export_state(self):
        return {k: getattr(self, k) for k in self._STATE_KEYS}

    def export_decode_view(self):
        return self.export_decode_view_from_state(self.export_state())

    @staticmethod
    def export_decode_view_from_state(state):
        keys = ('sign_mass_data', 'exp_data', 'invalid_exp', 'block_base', 'left', 'right', 'left_nbits', 'nbits',
                'blocksize', 'invalid_block_size', 'original_shape', 'n_elements', 'n_exp_data', 'device')
        return {k: state[k] for k in keys}

    @classmethod
    def from_state(cls, state):
        c = cls(right=state['right'], nbits=state['nbits'])
        for k in ('device', 'original_shape', 'n_elements', 'n_exp_data', 'sign_mass_data', 'exp_data',
                  'invalid_exp', 'block_base'):
            setattr(c, k, state[k])
        return c

    @classmethod
    def compress_block(cls, original_data_bfloat16, right, nbits, need_adjust=False):
        c = cls(right=right, nbits=nbits)
        hist = c.compress(original_data_bfloat16, need_adjust=need_adjust)
        return c, hist

    def materialize(self):
        return self.uncompress()

    # ------------------------------------------------------------------ pack
    def compress(self, original_data_bfloat16, need_adjust=False):
        """Pack the tensor (any shape, bf16, element count a multiple of 8); returns the int32[256]
        exponent histogram when ``need_adjust`` (reference: :768-822, :210-254)."""
        x = original_data_bfloat16
        if x.dtype != torch.bfloat16:
            raise ValueError(f'expected a bfloat16 tensor, got {x.dtype}')
        self.device = x.device
        self.original_shape = x.shape
        n = self.n_elements = x.numel()
        assert n % 8 == 0, 'the packed code plane holds whole groups of 8 elements'
        ibs = self.invalid_block_size
        flat = x.reshape(-1)
        if not flat.is_contiguous():
            flat = flat.contiguous()
        hist = torch.zeros(256, dtype=torch.int32, device=x.device) if need_adjust else None
        # one call; beyond _MAX_ELEMS_PER_CALL one per run of whole blocks
        per_call = max(ibs, (_MAX_ELEMS_PER_CALL // ibs) * ibs)
        signs, codes, escs, bases = [], [], [], []
        carried = 0
        for lo in range(0, n, per_call):
            sm, cd, esc, base = codec.pack_flat(flat[lo: lo + per_call], self.right, self.nbits, ibs, hist)
            signs.append(sm)
            codes.append(cd)
            escs.append(esc)
            bases.append(base + carried if carried else base)
            carried += esc.numel()
        self.sign_mass_data = signs[0] if len(signs) == 1 else torch.cat(signs)
        self.exp_data = codes[0] if len(codes) == 1 else torch.cat(codes)
        self.invalid_exp = escs[0] if len(escs) == 1 else torch.cat(escs)
        base = (bases[0] if len(bases) == 1 else torch.cat(bases)).to(torch.int32)
        self._base_i32 = base
        self.block_base = base.to(torch.int64)
        self.n_exp_data = n * self.nbits // 8
        return hist

    def _kernel_base(self) -> torch.Tensor:
        if self._base_i32 is None or self._base_i32.numel() != self.block_base.numel():
            self._base_i32 = self.block_base.to(torch.int32).contiguous()
        return self._base_i32

    # ------------------------------------------------------------------ unpack
    def uncompress_with_weights(self, uncompressed_odb):
        """Decode into ``uncompressed_odb`` (a flat 16-bit view of ``n_elements`` elements, bf16 or
        uint16/int16 storage; reference: :872-873)."""
        out = uncompressed_odb
        if out.numel() != self.n_elements or out.element_size() != 2 or not out.is_contiguous():
            raise ValueError('uncompress_with_weights needs a contiguous 16-bit buffer of n_elements elements')
        n = self.n_elements
        if n == 0:
            return
        dev = self.device
        sc = codec._scratch_for(dev)
        sm, cd, esc, dst = self.sign_mass_data, self.exp_data, self.invalid_exp, out
        if n < self.invalid_block_size:
            # (one short block may lie anywhere; the kernels want 16-byte boundaries)
            sm, cd = (t if t.data_ptr() % 16 == 0 else t.clone() for t in (sm, cd))
            if out.data_ptr() % 16:
                dst = torch.empty_like(out)
        with on_device(dev):
            rc = _lib.lib().adacode_unpack_flat_ragged(sm.data_ptr(), cd.data_ptr(), esc.data_ptr() if esc.numel() else 0, esc.numel(),
                                                       self._kernel_base().data_ptr(), n, self.left, self.nbits, dst.data_ptr(),
                                                       sc.status.data_ptr(), stream_ptr(dev))
        _lib.check(rc, 'adacode_unpack_flat_ragged')
        if dst is not out:
            out.copy_(dst)

    def uncompress(self):
        out = torch.empty(self.n_elements, dtype=torch.bfloat16, device=self.device)
        self.uncompress_with_weights(out)
        return out.view(self.original_shape)

    def update_compress(self, right, nbits):
        """Decode, forget the planes and adopt a new window (reference: :846-864)."""
        dense = self.uncompress()
        self.reset_memory()
        self._update_compression_params(right, nbits)
        return dense
