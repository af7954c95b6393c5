"""The flat layout at the ends of its blocks and tiles, against the oracle: sizes around one block and one tile of 16384,
short last blocks, windows over the lowest and highest exponents, streams that overflow the first guess, views off
16-byte boundaries."""
import numpy as np
import pytest
import torch

from tests import synth
from tests.test_flat_codec import _oracle_flat

pytestmark = pytest.mark.gpu


def _check(dev, x_cpu, right, nbits, out_shift=0):
    from adacode_b200 import codec
    from adacode_b200.compress_bitmap_merge import CompressorBitMap
    c = CompressorBitMap(right=right, nbits=nbits)
    hist = c.compress(x_cpu.to(dev), need_adjust=True)
    sm, cd, esc, base, want_hist = _oracle_flat(x_cpu, right, nbits, c.invalid_block_size)
    for name, got, want in (('signs', c.sign_mass_data, sm), ('codes', c.exp_data, cd), ('escapes', c.invalid_exp, esc),
                            ('base', c.block_base, base), ('hist', hist, want_hist)):
        assert np.array_equal(got.cpu().numpy(), want), name
    n = x_cpu.numel()
    room = torch.full((n + 32,), 77, dtype=torch.int16, device=dev)
    out = room[out_shift: out_shift + n]
    c.uncompress_with_weights(out)
    assert torch.equal(out.cpu(), x_cpu.view(torch.int16))
    assert (room[:out_shift] == 77).all() and (room[out_shift + n:] == 77).all()
    codec.check_device_status(dev)


@pytest.mark.parametrize('nbits', [1, 2, 3, 4])
@pytest.mark.parametrize('n', [8, 248, 256, 264, 504, 1016, 1024, 1032, 16384 - 8, 16384, 16384 + 8, 16384 + 1024 + 504, 5 * 16384 + 15 * 1024 + 1016,
                               4 * 2 ** 20 - 8, 4 * 2 ** 20, 4 * 2 ** 20 + 8, 4 * 2 ** 20 + 16384 + 15 * 1024 + 1016])
def test_sizes(cuda_device, n, nbits):
    x = synth.inject_escapes(synth.kv_tensor((1, 1, n // 8, 8), seed=n % 89, s=1.5), seed=4, left=121, right=128, p_window=0.05).reshape(-1)
    _check(cuda_device, x, 129, nbits)


@pytest.mark.parametrize('right,nbits', [(3, 3), (6, 3), (0, 1), (255, 2), (262, 3), (14, 4)])
def test_windows_at_the_ends_and_overflow(cuda_device, right, nbits):
    """All bf16 patterns and a short block behind them: nearly everything escapes, so the stream is packed again."""
    x = torch.cat([synth.all_bf16_patterns().reshape(-1), torch.zeros(120, dtype=torch.bfloat16)])
    _check(cuda_device, x, right, nbits)


def test_short_tensors_anywhere(cuda_device):
    x = synth.kv_tensor((1, 1, 12, 8), seed=5).reshape(-1)
    _check(cuda_device, x, 129, 3, out_shift=3)
    from adacode_b200.compress_bitmap_merge import CompressorBitMap
    room = torch.zeros(20000, dtype=torch.bfloat16, device=cuda_device)
    for n in (96, 1024, 1040, 2048, 16384, 16384 + 1032):
        view = room[5: 5 + n]
        view.copy_(synth.kv_tensor((1, 1, n // 8, 8), seed=6).reshape(-1))
        c = CompressorBitMap(129, 3)
        c.compress(view)
        assert torch.equal(c.uncompress().view(torch.int16), view.view(torch.int16))
