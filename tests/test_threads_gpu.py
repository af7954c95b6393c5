"""Packs and fused attention of several threads at a time: every byte is what one thread alone gets."""
import threading

import pytest
import torch

from tests import synth

pytestmark = pytest.mark.gpu

_PLANES = ('sign_mant', 'codes', 'escapes', 'tile_base', 'seg_offsets_dev')


def _all_at_once(device, work, n, own_streams):
    errors, start = [], threading.Barrier(n)

    def run(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream(device) if own_streams else torch.cuda.current_stream(device)):
                start.wait()
                for _ in range(25):
                    work(i)
        except BaseException as e:          # noqa: BLE001 (handed to the test's thread)
            errors.append(e)
    threads = [threading.Thread(target=run, args=(i,)) for i in range(n)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


# pipelined kernels, offsets scanned in the pack kernel (more than 65 536 tiles), direct kernels
@pytest.mark.parametrize('shape,seq_tile', [((1, 4, 1280, 64), 128), ((16, 64, 520, 16), 8), ((2, 3, 1280, 72), 128)])
@pytest.mark.parametrize('own_streams', [True, False])
def test_packs_do_not_share_a_scratch(cuda_device, shape, seq_tile, own_streams):
    from adacode_b200 import codec
    xs = [synth.kv_tensor(shape, seed=95 + i, s=0.5 + i).to(cuda_device) for i in range(4)]
    want = [codec.pack_blocks(x, 129, 3, seq_tile)[0] for x in xs]
    torch.cuda.synchronize(cuda_device)

    def work(i):
        got, _ = codec.pack_blocks(xs[i], 129, 3, seq_tile)
        out = torch.empty_like(xs[i])
        codec.unpack_chunk(got, out)
        assert torch.equal(out.view(torch.int16), xs[i].view(torch.int16))
        assert list(got.seg_offsets) == list(want[i].seg_offsets)
        for name in _PLANES:
            assert torch.equal(getattr(got, name), getattr(want[i], name)), name
    _all_at_once(cuda_device, work, len(xs), own_streams)
    codec.check_device_status(cuda_device)


# whole splits of a row, and runs that go on in the next row
@pytest.mark.parametrize('B,H,blocks', [(1, 8, 16), (32, 8, 5)])
@pytest.mark.parametrize('own_streams', [True, False])
def test_attention_does_not_share_partial_results(cuda_device, B, H, blocks, own_streams):
    from adacode_b200 import attention, codec
    calls = []
    for i in range(4):
        k, v = (synth.kv_tensor((B, H, 128 * blocks, 128), seed=s + i, s=0.5).to(cuda_device) for s in (60, 70))
        ks, vs = (codec.pack_blocks(x, 129, 3, 128)[0].segments() for x in (k, v))
        q = torch.randn(B, 4 * H, 128, generator=torch.Generator().manual_seed(i)).to(cuda_device, torch.bfloat16)
        calls.append((q, ks, vs, codec.build_segment_table(ks), codec.build_segment_table(vs)))

    def attend(i):
        q, ks, vs, kt, vt = calls[i]
        return attention.decode_attention(q, ks, vs, key_table=kt, value_table=vt)
    want = [attend(i) for i in range(4)]
    torch.cuda.synchronize(cuda_device)

    def work(i):
        got = [attend(i) for _ in range(4)]
        for g in got:
            assert torch.equal(g.view(torch.int16), want[i].view(torch.int16))
    _all_at_once(cuda_device, work, 4, own_streams)
    codec.check_device_status(cuda_device)
