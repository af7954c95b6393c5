"""Edges of the decode in registers (unpack and fused attention) and of the exponent histogram: escapes beyond
the staged part of a tile's stream, every code length, rows that are not 32-byte aligned, views of every
stride order."""
import math

import numpy as np
import pytest
import torch

from tests import synth

pytestmark = pytest.mark.gpu


def _bits(t):
    return t.contiguous().view(torch.int16)


@pytest.mark.parametrize('nbits', [1, 2, 3, 4])
@pytest.mark.parametrize('shape', [(1, 2, 256, 128), (2, 1, 128, 64), (1, 1, 128, 80), (1, 1, 128, 512), (1, 1, 16, 2048)])
@pytest.mark.parametrize('share', [0.0, 0.3, 1.0])
def test_unpack_any_share_of_escapes(cuda_device, nbits, shape, share):
    """``share`` of the elements outside the window (1: all of them, more than a stage holds)."""
    from adacode_b200 import codec
    right = 130
    g = torch.Generator('cpu').manual_seed(nbits * 100 + shape[3])
    e = torch.randint(right - 2 ** nbits + 2, right + 1, shape, generator=g)
    out_e = torch.randint(0, 2, shape, generator=g) * 255        # 0 and 255: the ends of the byte
    e = torch.where(torch.rand(shape, generator=g) < share, out_e, e)
    raw = (e << 7) | torch.randint(0, 128, shape, generator=g) | (torch.randint(0, 2, shape, generator=g) << 15)
    x = raw.to(torch.int32).to(torch.int16).view(torch.bfloat16).to(cuda_device)
    tile = min(128, shape[2])
    chunk, _ = codec.pack_blocks(x, right, nbits, tile)
    out = torch.zeros_like(x)
    codec.unpack_chunk(chunk, out)
    assert torch.equal(_bits(out), _bits(x))
    # rows of a longer buffer that start on 16-byte but not on 32-byte boundaries
    wide = torch.zeros(shape[0], shape[1], shape[2], shape[3] + 8, dtype=torch.bfloat16, device=cuda_device)
    codec.unpack_segments(chunk.segments(), wide[..., 8:])
    assert torch.equal(_bits(wide[..., 8:]), _bits(x)) and int(_bits(wide[..., :8]).abs().max()) == 0
    codec.check_device_status(cuda_device)


@pytest.mark.parametrize('D', [64, 128])
@pytest.mark.parametrize('G', [1, 8, 9, 16, 17])
@pytest.mark.parametrize('params', [(130, 3), (100, 1), (126, 4)])
def test_attention_beyond_the_window(cuda_device, D, G, params):
    """(100, 1): every element escapes.  Compared with 64-bit attention: the result is rounded to bf16 (2**-9) and
    probabilities keep at least 17 bits, so twice the rounding bounds the error."""
    from adacode_b200 import attention, codec
    S, tail = 256 + 41, 41
    k = synth.kv_tensor((1, 2, S, D), seed=7, key_offset=True, s=0.5).to(cuda_device)
    v = synth.kv_tensor((1, 2, S, D), seed=8, s=0.5).to(cuda_device)
    q = (0.5 * torch.randn(1, 2 * G, D, generator=torch.Generator('cpu').manual_seed(G))).to(torch.bfloat16).to(cuda_device)
    ks = codec.pack_blocks(k[:, :, :S - tail], *params, 128)[0].segments()
    vs = codec.pack_blocks(v[:, :, :S - tail], *params, 128)[0].segments()
    # a tail whose rows lie on 4-byte boundaries only
    buf = torch.zeros(2, 1, 2, tail, D + 2, dtype=torch.bfloat16, device=cuda_device)
    buf[0, ..., 2:], buf[1, ..., 2:] = k[:, :, S - tail:], v[:, :, S - tail:]
    for kt, vt in ((k[:, :, S - tail:], v[:, :, S - tail:]), (buf[0][..., 2:], buf[1][..., 2:])):
        out = attention.decode_attention(q, ks, vs, kt, vt, n_splits=2).double()
        p = torch.softmax(q.view(1, 2, G, D).double() @ k.double().transpose(-1, -2) / math.sqrt(D), dim=-1)
        ref = (p @ v.double()).view(1, 2 * G, D)
        scale = (p @ v.double().abs()).view(1, 2 * G, D)         # what the sums' rounding is relative to
        assert ((out - ref).abs() <= 2.0 ** -8 * ref.abs() + 2.0 ** -14 * scale).all()
    codec.check_device_status(cuda_device)


@pytest.mark.parametrize('shape', [(1, 1, 1, 8), (1, 1, 1, 1024), (1, 1, 3, 1032), (2, 3, 5, 72), (2, 4, 128, 128), (1, 8, 33, 512), (3, 2, 300, 64)])
def test_histogram_of_any_view(cuda_device, shape):
    """Against a count on the CPU: contiguous, projections seen as [B, H, S, D], slices of a longer buffer, dimensions
    in every order, expanded ones."""
    from adacode_b200 import codec
    B, H, S, D = shape
    g = torch.Generator('cpu').manual_seed(S * D)
    raw = torch.randint(-2 ** 15, 2 ** 15, (B, H, S, D), generator=g).to(torch.int16)
    raw[..., ::2] = (raw[..., ::2] & ~0x7F80) | (124 << 7)        # most lanes in one bin
    x = raw.view(torch.bfloat16).to(cuda_device)
    longer = torch.zeros(B, H, S + 7, D, dtype=torch.bfloat16, device=cuda_device)
    longer[:, :, 3:3 + S] = x
    views = [x, longer[:, :, 3:3 + S], x[:1].expand(3, H, S, D), x.permute(1, 0, 2, 3)]
    views += [x.permute(*order, 3).contiguous().permute(*[order.index(i) for i in range(3)], 3) for order in ((0, 2, 1), (2, 1, 0), (1, 0, 2))]
    for t in views:
        got = codec.exponent_hist(t).cpu().numpy()
        e = (t.contiguous().view(torch.int16).cpu().numpy().astype(np.int64) >> 7) & 0xFF
        assert np.array_equal(got, np.bincount(e.ravel(), minlength=256))


@pytest.mark.parametrize('B,H,blocks,D', [(1, 1, 1, 128), (1, 3, 1, 64), (3, 1, 333, 16), (1, 5, 2400, 16), (2, 4, 8193, 16)])
def test_offsets_of_many_tiles(cuda_device, B, H, blocks, D):
    """Escape offsets of two tensors of one launch, from one tile up to 131 088 (two tensors of 65 544 tiles: beyond what
    the compaction's CTAs add up themselves), against sums of the tiles' own counts; then the round trip."""
    from adacode_b200 import codec
    g = torch.Generator(device=cuda_device).manual_seed(blocks)
    k, v = (torch.randn(B, H, blocks * 128, D, generator=g, device=cuda_device).to(torch.bfloat16) for _ in range(2))
    chunks = codec.pack_pair(k, v, (127, 3), (126, 3), 128)[:2]
    for x, c, right in zip((k, v), chunks, (127, 126)):
        e = (x.view(torch.int16).to(torch.int32) >> 7) & 0xFF
        out = ((e <= right - 7) | (e > right)).view(B, H, blocks, 128 * D).sum(-1).permute(2, 0, 1).reshape(blocks, B * H)
        assert torch.equal(c.tile_base.long(), out.cumsum(1))
        assert torch.equal(c.seg_offsets_dev, torch.cat([torch.zeros_like(out[:1, 0]), out.sum(1).cumsum(0)]))
        back = torch.empty_like(x)
        codec.unpack_chunk(c, back)
        assert torch.equal(_bits(back), _bits(x))
    codec.check_device_status(cuda_device)
