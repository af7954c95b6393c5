"""Packs of several threads at a time: every byte is what one thread alone gets, and unpacks to the input."""
import threading

import pytest
import torch

from tests import synth

pytestmark = pytest.mark.gpu

_PLANES = ('sign_mant', 'codes', 'escapes', 'tile_base', 'seg_offsets_dev')


# pipelined kernels, offsets scanned in the pack kernel (more than 65 536 tiles), direct kernels
@pytest.mark.parametrize('shape,seq_tile', [((1, 4, 1280, 64), 128), ((16, 64, 520, 16), 8), ((2, 3, 1280, 72), 128)])
@pytest.mark.parametrize('own_streams', [True, False])
def test_packs_do_not_share_a_scratch(cuda_device, shape, seq_tile, own_streams):
    from adacode_b200 import codec
    xs = [synth.kv_tensor(shape, seed=95 + i, s=0.5 + i).to(cuda_device) for i in range(4)]
    want = [codec.pack_blocks(x, 129, 3, seq_tile)[0] for x in xs]
    torch.cuda.synchronize(cuda_device)
    errors, start = [], threading.Barrier(len(xs))

    def work(i):
        try:
            stream = torch.cuda.Stream(cuda_device) if own_streams else torch.cuda.current_stream(cuda_device)
            with torch.cuda.stream(stream):
                start.wait()
                for _ in range(25):
                    got, _ = codec.pack_blocks(xs[i], 129, 3, seq_tile)
                    out = torch.empty_like(xs[i])
                    codec.unpack_chunk(got, out)
                    assert torch.equal(out.view(torch.int16), xs[i].view(torch.int16))
                    assert list(got.seg_offsets) == list(want[i].seg_offsets)
                    for name in _PLANES:
                        assert torch.equal(getattr(got, name), getattr(want[i], name)), name
        except BaseException as e:          # noqa: BLE001 (handed to the test's thread)
            errors.append(e)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(xs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    codec.check_device_status(cuda_device)
