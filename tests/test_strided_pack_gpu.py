"""Pack of sources whose token rows do not follow each other (one tensor copy per unit, or row copies where a box cannot
describe the unit) against the pack of a contiguous copy, byte for byte, and the round trip."""
import pytest
import torch

from tests import synth

pytestmark = pytest.mark.gpu


def _bshd(shape, dev):
    B, H, S, D = shape
    return synth.kv_tensor((B, S, H, D), seed=5, key_offset=True).to(dev).transpose(1, 2)


def _sbhd(shape, dev):
    B, H, S, D = shape
    return synth.kv_tensor((S, B, H, D), seed=6, key_offset=True).to(dev).permute(1, 2, 0, 3)


def _wide_rows(shape, dev):
    B, H, S, D = shape
    return synth.kv_tensor((B, H, S, D + 24), seed=7, key_offset=True).to(dev)[..., 16:16 + D]


def _every_other_token(shape, dev):
    B, H, S, D = shape
    return synth.kv_tensor((B, H, 2 * S, D), seed=8, key_offset=True).to(dev)[:, :, 1::2]


def _one_head_for_all(shape, dev):
    B, H, S, D = shape
    return _wide_rows((B, 1, S, D), dev).expand(B, H, S, D)


def _one_token_for_all(shape, dev):
    B, H, S, D = shape
    return synth.kv_tensor((B, H, 1, D), seed=9, key_offset=True).to(dev).expand(B, H, S, D)


_SOURCES = [_bshd, _sbhd, _wide_rows, _every_other_token, _one_head_for_all, _one_token_for_all]


# tiles of one whole unit, of several, of a last unit with fewer rows; more than 256 rows or 1024 columns: row copies
@pytest.mark.parametrize('shape,seq_tile', [((2, 3, 256, 128), 128), ((1, 8, 384, 64), 128), ((3, 1, 128, 1024), 128),
                                            ((2, 2, 128, 1040), 128), ((2, 2, 720, 96), 240), ((1, 2, 1024, 16), 512),
                                            ((2, 1, 48, 512), 24), ((1, 5, 16, 272), 8), ((1, 1, 256, 128), 256)])
@pytest.mark.parametrize('source', _SOURCES, ids=lambda f: f.__name__[1:])
def test_strided_source_packs_like_its_copy(cuda_device, source, shape, seq_tile):
    from adacode_b200 import codec
    x = source(shape, cuda_device)
    assert tuple(x.shape) == shape
    for nbits in (2, 3):
        got, hist = codec.pack_blocks(x, 129, nbits, seq_tile, need_hist=True)
        want, want_hist = codec.pack_blocks(x.contiguous(), 129, nbits, seq_tile, need_hist=True)
        for field in ('sign_mant', 'codes', 'escapes', 'tile_base', 'seg_offsets_dev'):
            assert torch.equal(getattr(got, field), getattr(want, field)), field
        assert torch.equal(hist, want_hist)
        out = torch.empty(shape, dtype=torch.bfloat16, device=cuda_device)
        codec.unpack_chunk(got, out)
        assert torch.equal(out.view(torch.int16), x.contiguous().view(torch.int16))
    codec.check_device_status(cuda_device)


def test_strided_jobs_of_one_launch(cuda_device):
    """Keys strided, values contiguous, in one launch."""
    from adacode_b200 import codec
    k, v = _bshd((2, 4, 384, 128), cuda_device), synth.kv_tensor((2, 4, 384, 128), seed=10).to(cuda_device)
    kc, vc, *_ = codec.pack_pair(k, v, (130, 3), (128, 3), 128)
    for chunk, x in ((kc, k), (vc, v)):
        out = torch.empty(2, 4, 384, 128, dtype=torch.bfloat16, device=cuda_device)
        codec.unpack_chunk(chunk, out)
        assert torch.equal(out.view(torch.int16), x.contiguous().view(torch.int16))
    codec.check_device_status(cuda_device)
