"""Device memory that the escapes of a packed span hold on to."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('nbits', [1, 2])
@pytest.mark.parametrize('blocks', [1, 3, 40])
@pytest.mark.parametrize('share', [0.0, 0.1, 0.3])
def test_first_guess_is_cut_to_size(cuda_device, nbits, blocks, share):
    """Packed without a known share: at most an eighth more than the escapes, and a 32nd of the elements, stay allocated
    (one block of [1, 8, 128, 128] at 10 % escapes and two bits: 13 KB of 131 072, not the 64 KB guessed)."""
    from adacode_b200 import codec
    g = torch.Generator('cpu').manual_seed(blocks)
    shape = (1, 8, 128 * blocks, 128)
    e = torch.where(torch.rand(shape, generator=g) < share, 100, 130)
    x = ((e << 7) | torch.randint(0, 128, shape, generator=g)).to(torch.int16).view(torch.bfloat16).to(cuda_device)
    chunk, _ = codec.pack_blocks(x, 130, nbits, 128)
    other, _, *_ = codec.pack_pair(x, x, (130, nbits), (130, nbits), 128)
    for c in (chunk, other):
        n = c.escapes.numel()
        assert n == int((e == 100).sum())
        assert c.escapes.untyped_storage().nbytes() <= n + n // 8 + min(65536, x.numel() // 32)
        out = torch.empty_like(x)
        codec.unpack_chunk(c, out)
        assert torch.equal(out.view(torch.int16), x.view(torch.int16))
