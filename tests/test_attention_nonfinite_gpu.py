"""Infinities and NaN in the query, the keys and the values of fused attention: an output entry is finite, infinite
or NaN where 64-bit attention has it so, and the finite ones keep their precision."""
import math

import pytest
import torch

from tests import synth

pytestmark = pytest.mark.gpu

INF, NAN = float('inf'), float('nan')
PACKED, TAIL = 256, 41                     # tokens; the tail starts at 256


def _put(t, where, entries):
    """Entries {(token, column): value} of head 1, the tokens counted from the start of the packed or the dense part."""
    for (token, col), value in entries.items():
        t[0, 1, token + (PACKED if where == 'tail' else 0), col] = value


def _check(dev, D, G, n_splits, q, k, v):
    from adacode_b200 import attention, codec
    q, k, v = q.to(dev), k.to(dev), v.to(dev)
    ks = codec.pack_blocks(k[:, :, :PACKED], 130, 3, 128)[0].segments()
    vs = codec.pack_blocks(v[:, :, :PACKED], 127, 3, 128)[0].segments()
    out = attention.decode_attention(q, ks, vs, k[:, :, PACKED:], v[:, :, PACKED:], n_splits=n_splits).double()
    codec.check_device_status(dev)
    p = torch.softmax(q.view(1, 2, G, D).double() @ k.double().transpose(-1, -2) / math.sqrt(D), dim=-1)
    ref = (p @ v.double()).view(1, 2 * G, D)
    scale = (p @ v.double().abs()).view(1, 2 * G, D)
    assert torch.equal(out.isnan(), ref.isnan())
    assert torch.equal(out == INF, ref == INF) and torch.equal(out == -INF, ref == -INF)
    fin = ref.isfinite()
    assert ((out - ref).abs() <= 2.0 ** -8 * ref.abs() + 2.0 ** -14 * scale)[fin].all()      # (as with finite inputs)
    return fin


def _inputs(D, G):
    S = PACKED + TAIL
    k, v = synth.kv_tensor((1, 2, S, D), seed=17, s=0.3), synth.kv_tensor((1, 2, S, D), seed=18, s=0.5)
    q = (0.5 * torch.randn(1, 2 * G, D, generator=torch.Generator('cpu').manual_seed(G))).to(torch.bfloat16)
    return q, k, v


@pytest.mark.parametrize('D', [64, 128])
@pytest.mark.parametrize('G', [1, 9])
@pytest.mark.parametrize('n_splits', [1, 3, 17])
@pytest.mark.parametrize('where', ['packed', 'tail'])
def test_scores(cuda_device, D, G, n_splits, where):
    """A NaN in a key makes its head NaN, an infinite key decides by the query's sign (weight 0, or NaN for all), a
    NaN or an infinity in a query concerns that query alone."""
    q, k, v = _inputs(D, G)
    for value in (NAN, INF, -INF):
        kx = k.clone()
        _put(kx, where, {(7, 5): value})
        _check(cuda_device, D, G, n_splits, q, kx, v)
        qx = q.clone()
        qx[0, G, 3] = value
        fin = _check(cuda_device, D, G, n_splits, qx, k, v)
        assert not fin[0, G].any() and fin[0, :G].all() and fin[0, G + 1:].all()


@pytest.mark.parametrize('D', [64, 128])
@pytest.mark.parametrize('G', [1, 9])
@pytest.mark.parametrize('n_splits', [1, 3, 17])
@pytest.mark.parametrize('where', ['packed', 'tail'])
def test_values(cuda_device, D, G, n_splits, where):
    """An infinite value makes its column infinite whatever its token's weight, infinities of both signs or a NaN make
    it NaN; the other columns keep the precision that they have with finite values."""
    q, k, v = _inputs(D, G)
    at = PACKED if where == 'tail' else 0
    last = D - 1
    v[0, 1, at: at + 41, 12] = INF                              # every token of the tail, or a third of a block
    _put(v, where, {(0, 0): INF, (40, 3): -INF, (7, 5): NAN, (9, 9): INF, (33, 9): -INF, (21, last): INF, (22, last): INF})
    fin = _check(cuda_device, D, G, n_splits, q, k, v)
    assert fin[0, :G].all() and int((~fin[0, G]).sum()) == 6
    # ... one token has all the weight (a probability of exactly 1, nothing left over for the further terms)
    one = torch.zeros_like(k)
    one[0, :, at + 21] = 8 * q[0, ::G].sign()
    one[0, :, at + 21][..., 1::2] = 0
    _check(cuda_device, D, G, n_splits, q[:, ::G].repeat_interleave(G, 1), one, v)


@pytest.mark.parametrize('D', [64, 128])
def test_values_over_many_blocks(cuda_device, D):
    """Units of the second walk follow those of the first in the same ring: 21 blocks in one CTA, windows and code lengths
    alternating, infinities in the first, a middle and the last one."""
    from adacode_b200 import attention, codec
    S, G = 21 * 128, 4
    k, v = synth.kv_tensor((1, 2, S, D), seed=27, s=0.3), synth.kv_tensor((1, 2, S, D), seed=28, s=0.5)
    q = (0.5 * torch.randn(1, 2 * G, D, generator=torch.Generator('cpu').manual_seed(3))).to(torch.bfloat16)
    v[0, 0, 5, 1], v[0, 0, 1300, 2], v[0, 0, S - 1, 3], v[0, 0, 200, 4], v[0, 0, 2000, 4] = INF, -INF, INF, INF, -INF
    q, k, v = q.to(cuda_device), k.to(cuda_device), v.to(cuda_device)
    segs = [[codec.pack_blocks(t[:, :, i: i + 128], *((130, 3), (127, 4), (126, 2), (124, 1))[i // 128 % 4], 128)[0].segment(0)
             for i in range(0, S, 128)] for t in (k, v)]
    out = attention.decode_attention(q, *segs, n_splits=1).double()
    codec.check_device_status(cuda_device)
    p = torch.softmax(q.view(1, 2, G, D).double() @ k.double().transpose(-1, -2) / math.sqrt(D), dim=-1)
    ref = (p @ v.double()).view(1, 2 * G, D)
    scale = (p @ v.double().abs()).view(1, 2 * G, D)
    assert torch.equal(out.isnan(), ref.isnan()) and torch.equal(out[out.isinf()], ref[out.isinf()])
    fin = ref.isfinite()
    assert torch.equal(fin, out.isfinite()) and int((~fin).sum()) == 4 * G
    assert ((out - ref).abs() <= 2.0 ** -8 * ref.abs() + 2.0 ** -14 * scale)[fin].all()
