"""The pack that reports to the host: what it sends is what the device buffer holds, for the pipelined kernels with one
compaction CTA and with many, with the escape offsets scanned by the pack kernel, and for the direct kernels."""
import ctypes

import pytest
import torch

from tests import synth

pytestmark = pytest.mark.gpu


# one tile; several; more tiles than the compaction's CTAs add up (65 536); head sizes of the direct kernels (72, 8)
@pytest.mark.parametrize('shape,seq_tile', [((1, 1, 128, 128), 128), ((3, 5, 640, 64), 128), ((16, 64, 520, 16), 8), ((2, 3, 256, 72), 128),
                                            ((1, 2, 128, 8), 128)])
def test_report_is_what_the_device_holds(cuda_device, shape, seq_tile):
    from adacode_b200 import codec
    k = synth.kv_tensor(shape, seed=71, key_offset=True).to(cuda_device)
    v = synth.kv_tensor(shape, seed=72).to(cuda_device)
    for turn in range(3):                          # the scratch's counters are left as they were found
        kc, vc, kh, vh, kh_host, vh_host = codec.pack_pair(k, v, (130, 3), (127, 3), seq_tile, need_hist=True)
        for x, c, h, h_host, right in ((k, kc, kh, kh_host, 130), (v, vc, vh, vh_host, 127)):
            assert c.seg_offsets_dev.cpu().tolist() == list(c.seg_offsets)
            assert torch.equal(h.cpu(), torch.from_numpy(h_host))
            assert int(h_host.sum()) == x.numel()
            one, _ = codec.pack_blocks(x, right, 3, seq_tile)
            assert list(one.seg_offsets) == list(c.seg_offsets) and torch.equal(one.escapes, c.escapes)
            out = torch.empty_like(x)
            codec.unpack_chunk(c, out)
            assert torch.equal(out.view(torch.int16), x.view(torch.int16))
    codec.check_device_status(cuda_device)


def test_reports_of_different_lengths_and_streams(cuda_device):
    """A token may lie where an earlier, longer report had data; packs on a side stream report as well."""
    from adacode_b200 import codec
    x = synth.kv_tensor((1, 2, 128 * 40, 64), seed=73).to(cuda_device)
    side = torch.cuda.Stream(cuda_device)
    side.wait_stream(torch.cuda.current_stream(cuda_device))
    for blocks in (40, 1, 7, 2, 39):
        want, _ = codec.pack_blocks(x[:, :, :128 * blocks], 129, 3, 128)
        with torch.cuda.stream(side):
            got, _ = codec.pack_blocks(x[:, :, :128 * blocks], 129, 3, 128)
        assert list(got.seg_offsets) == list(want.seg_offsets)
        assert got.seg_offsets_dev.cpu().tolist() == list(want.seg_offsets)
    torch.cuda.current_stream(cuda_device).wait_stream(side)


@pytest.mark.parametrize('blocks', [1, 40])
def test_the_host_may_go_on_from_any_stream(cuda_device, blocks):
    """A pack that has returned has written its outputs and is done with its scratch: other streams need not wait for it."""
    from adacode_b200 import codec
    x = synth.kv_tensor((1, 4, 128 * blocks, 128), seed=74).to(cuda_device)
    want, _ = codec.pack_blocks(x, 129, 3, 128)
    torch.cuda.synchronize(cuda_device)
    streams = [torch.cuda.Stream(cuda_device) for _ in range(3)]
    for turn in range(40):
        with torch.cuda.stream(streams[turn % 3]):
            got, _ = codec.pack_blocks(x, 129, 3, 128)
        with torch.cuda.stream(streams[(turn + 1) % 3]):
            out = torch.empty_like(x)
            codec.unpack_chunk(got, out)
            assert torch.equal(out.view(torch.int16), x.view(torch.int16))
            for name in ('sign_mant', 'codes', 'escapes', 'tile_base', 'seg_offsets_dev'):
                assert torch.equal(getattr(got, name), getattr(want, name)), name


def test_refusals(cuda_device):
    from adacode_b200 import _lib
    L = _lib.lib()
    dev = torch.zeros(64, dtype=torch.uint8, device=cuda_device)
    pinned = torch.zeros(128, dtype=torch.uint8).pin_memory()
    jobs = (_lib.PackJob * 1)()

    def call(report, host, nbytes):
        return L.adacode_pack_jobs_report(ctypes.addressof(jobs), 0, 1, 1, 128, 128, 3, None, 0, dev.data_ptr(), report, host, nbytes, 1,
                                          torch.cuda.current_stream().cuda_stream)
    assert call(dev.data_ptr(), pinned.data_ptr(), 6) == _lib.ERR_INVALID_ARG
    assert call(dev.data_ptr() + 2, pinned.data_ptr(), 8) == _lib.ERR_INVALID_ARG
    assert call(dev.data_ptr(), pinned.data_ptr() + 4, 8) == _lib.ERR_INVALID_ARG
    assert call(dev.data_ptr(), torch.zeros(128, dtype=torch.uint8).data_ptr(), 8) == _lib.ERR_INVALID_ARG      # not page-locked
    assert call(dev.data_ptr(), pinned.data_ptr(), (1 << 20) + 4) == _lib.ERR_TOO_LARGE
    assert call(dev.data_ptr(), pinned.data_ptr(), 8) == _lib.OK                                            # no jobs: the cleared words
    out = torch.full((2,), -1, dtype=torch.int32)
    stream = torch.cuda.current_stream().cuda_stream
    assert L.adacode_wait_report(pinned.data_ptr(), 8, 1, out.data_ptr(), stream) == _lib.OK and not out.any()
    # a token that nothing will send: an error as soon as the stream is idle
    assert L.adacode_wait_report(pinned.data_ptr(), 8, 77, out.data_ptr(), stream) == _lib.ERR_CUDA
