"""Fused attention whose work is cut through all rows (batch, KV head, group of query heads): runs that begin and end in
the middle of a row, cover whole rows, or lie in the dense tail alone."""
import math

import pytest
import torch

from tests import synth

pytestmark = pytest.mark.gpu


def _inputs(dev, B, Hkv, G, D, n_seg, tail):
    from adacode_b200 import codec
    S = n_seg * 128 + tail
    k = synth.kv_tensor((B, Hkv, S, D), seed=61, key_offset=True, s=0.5).to(dev)
    v = synth.kv_tensor((B, Hkv, S, D), seed=62, s=0.5).to(dev)
    q = (0.5 * torch.randn(B, Hkv * G, D, generator=torch.Generator('cpu').manual_seed(G))).to(torch.bfloat16).to(dev)
    ks, vs = ([codec.pack_blocks(t[:, :, 128 * j: 128 * (j + 1)], 130 - j % 3, 2 + (j + o) % 3, 128)[0].segment(0) for j in range(n_seg)]
              for t, o in ((k, 0), (v, 1)))
    return q, k, v, ks, vs


def _check(out, q, k, v):
    """One rounding to bf16 (2**-9) and at least 17 bits of every probability: twice the rounding bounds the error."""
    (B, Hkv, S, D), out = k.shape, out.double()
    p = torch.softmax(q.view(B, Hkv, -1, D).double() @ k.double().transpose(-1, -2) / math.sqrt(D), dim=-1)
    ref, scale = (p @ v.double()).view(q.shape), (p @ v.double().abs()).view(q.shape)
    assert ((out - ref).abs() <= 2.0 ** -8 * ref.abs() + 2.0 ** -14 * scale).all()


# more rows than CTAs with one item each and with several; items of which most or all are dense; two groups of heads
@pytest.mark.parametrize('B,Hkv,G,D,n_seg,tail', [(300, 1, 4, 64, 1, 0), (101, 3, 4, 128, 2, 30), (37, 4, 20, 128, 2, 0),
                                                  (150, 2, 1, 128, 1, 300), (307, 1, 8, 64, 0, 290), (8, 4, 7, 128, 11, 5),
                                                  (43, 7, 16, 64, 3, 1), (5, 4, 9, 128, 20, 129)])
def test_runs_across_rows(cuda_device, B, Hkv, G, D, n_seg, tail):
    from adacode_b200 import attention, codec
    q, k, v, ks, vs = _inputs(cuda_device, B, Hkv, G, D, n_seg, tail)
    kt, vt = (k[:, :, n_seg * 128:], v[:, :, n_seg * 128:]) if tail else (None, None)
    for n_splits in (0, 2):
        _check(attention.decode_attention(q, ks, vs, kt, vt, n_splits=n_splits), q, k, v)
    codec.check_device_status(cuda_device)


def test_workspace_for_whole_splits_only(cuda_device):
    """256 rows of 16 blocks: one split each asks for less workspace than one cut through all of them, and is taken where
    the workspace holds no more; less than that is refused."""
    from adacode_b200 import _lib, codec
    B, Hkv, G, D = 64, 4, 1, 64
    q, k, v, ks, vs = _inputs(cuda_device, B, Hkv, G, D, 16, 0)
    L, kt, vt = _lib.lib(), codec.build_segment_table(ks), codec.build_segment_table(vs)
    status, out = torch.zeros(2, dtype=torch.int32, device=cuda_device), torch.empty_like(q)
    one = int(L.adacode_decode_attn_workspace_bytes(B, Hkv * G, D, 1))
    ws = torch.full((one + 4096,), 0xA5, dtype=torch.uint8, device=cuda_device)

    def call(nbytes):
        return L.adacode_decode_attn(q.data_ptr(), q.stride(0), q.stride(1), kt.data_ptr(), vt.data_ptr(), 16, None, None, 0, 0, 0, 0,
                                     B, Hkv * G, Hkv, 128, D, D ** -0.5, out.data_ptr(), ws.data_ptr(), nbytes, 0, status.data_ptr(),
                                     torch.cuda.current_stream().cuda_stream)
    assert call(one - 1) == _lib.ERR_WORKSPACE
    assert call(one) == _lib.OK
    _check(out, q, k, v)
    assert (ws[one:] == 0xA5).all() and int(status[0]) == 0
