"""Fused attention over many blocks: rings that wrap, source tables that are looked up again every 32 units, windows
and code lengths that change from block to block, and the combine kernel over few and many splits, empty ones
among them."""
import math

import pytest
import torch

from tests import synth

pytestmark = pytest.mark.gpu

_WINDOWS = ((130, 3), (129, 4), (128, 2), (127, 3), (126, 1))


@pytest.fixture(scope='module')
def packed(cuda_device):
    """Per head size: keys and values of 40 blocks and 200 further tokens, and their segments (five windows in turn)."""
    from adacode_b200 import codec
    out = {}
    for D in (64, 128):
        k = synth.kv_tensor((1, 2, 40 * 128 + 200, D), seed=41, key_offset=True, s=0.5).to(cuda_device)
        v = synth.kv_tensor((1, 2, 40 * 128 + 200, D), seed=42, s=0.5).to(cuda_device)
        segs = [[codec.pack_blocks(t[:, :, 128 * j: 128 * (j + 1)], *_WINDOWS[(j + o) % 5], 128)[0].segment(0) for j in range(40)]
                for t, o in ((k, 0), (v, 2))]
        out[D] = (k, v, *segs)
    return out


@pytest.mark.parametrize('D', [64, 128])
@pytest.mark.parametrize('G', [4, 16])
@pytest.mark.parametrize('n_splits', [1, 2, 16, 17, 33, 128])
@pytest.mark.parametrize('tail', [0, 200])
def test_forty_blocks(cuda_device, packed, D, G, n_splits, tail):
    """1: 80 units in one CTA, two of whose table lookups are later ones; 16 and 17: both sides of the combine kernel's
    rule; 128: most splits have nothing.  Compared with 64-bit attention: one rounding to bf16 (2**-9) and at least
    17 bits of every probability, so twice the rounding bounds the error."""
    from adacode_b200 import attention, codec
    k, v, ks, vs = packed[D]
    S = 40 * 128 + tail
    q = (0.5 * torch.randn(1, 2 * G, D, generator=torch.Generator('cpu').manual_seed(G))).to(torch.bfloat16).to(cuda_device)
    kt, vt = (k[:, :, 5120:S], v[:, :, 5120:S]) if tail else (None, None)
    out = attention.decode_attention(q, ks, vs, kt, vt, n_splits=n_splits).double()
    codec.check_device_status(cuda_device)
    p = torch.softmax(q.view(1, 2, G, D).double() @ k[:, :, :S].double().transpose(-1, -2) / math.sqrt(D), dim=-1)
    ref = (p @ v[:, :, :S].double()).view(1, 2 * G, D)
    scale = (p @ v[:, :, :S].double().abs()).view(1, 2 * G, D)
    assert ((out - ref).abs() <= 2.0 ** -8 * ref.abs() + 2.0 ** -14 * scale).all()
