"""The extension module behind packs and decode steps: what it leaves to the calls from Python (modes, subclasses, gradients),
launches of unequal tensors, reports too long for pinned memory, overflow, threads."""
import threading

import pytest
import torch
from torch.overrides import TorchFunctionMode

from tests import synth
from tests.scenarios import StubConfig

pytestmark = pytest.mark.gpu


def _round_trip(chunk, x):
    from adacode_b200 import codec
    out = torch.empty(x.shape, dtype=x.dtype, device=x.device)
    codec.unpack_chunk(chunk, out)
    assert torch.equal(out.view(torch.int16), x.contiguous().view(torch.int16))
    assert chunk.seg_offsets_dev.cpu().tolist() == list(chunk.seg_offsets) and chunk.escapes.numel() == chunk.seg_offsets[-1]


@pytest.mark.parametrize('ks,vs,kp,vp', [((2, 3, 256, 128), (2, 3, 256, 64), (130, 3), (127, 3)),     # two head sizes
                                         ((1, 2, 384, 64), (1, 2, 384, 64), (130, 3), (127, 4)),      # two code lengths
                                         ((1, 2, 256, 72), (1, 2, 256, 72), (130, 2), (127, 2)),      # the direct kernels
                                         ((1, 2, 0, 64), (1, 2, 0, 64), (130, 3), (127, 3))])         # nothing to pack
@pytest.mark.parametrize('capacity', [None, 5])                                                       # 5: overflows, packed again
def test_pairs(cuda_device, ks, vs, kp, vp, capacity):
    from adacode_b200 import codec
    k, v = synth.kv_tensor(ks, seed=81, key_offset=True).to(cuda_device), synth.kv_tensor(vs, seed=82).to(cuda_device)
    kc, vc, kh, vh, khh, vhh = codec.pack_pair(k, v, kp, vp, 128, need_hist=True, capacities=(capacity, capacity))
    for x, c, h, hh in ((k, kc, kh, khh), (v, vc, vh, vhh)):
        want = torch.bincount((x.reshape(-1).view(torch.int16).int() >> 7) & 0xFF, minlength=256)
        assert torch.equal(h.long(), want) and torch.equal(torch.from_numpy(hh).long(), want.cpu())
        _round_trip(c, x)
    codec.check_device_status(cuda_device)


def test_histogram_that_is_added_to(cuda_device):
    from adacode_b200 import codec
    x = synth.kv_tensor((1, 2, 256, 64), seed=83).to(cuda_device)
    hist = torch.full((256,), 7, dtype=torch.int32, device=cuda_device)
    chunk, got = codec.pack_blocks(x, 129, 3, 128, need_hist=True, hist_out=hist)
    assert got is hist and int(hist.sum()) == 7 * 256 + x.numel()
    _round_trip(chunk, x)


def test_more_offsets_than_a_report_holds(cuda_device):
    """140 000 blocks of eight tokens: 1.1 MB of offsets, fetched by a copy."""
    from adacode_b200 import codec
    x = synth.kv_tensor((1, 1, 8 * 140_000, 16), seed=84).to(cuda_device)
    chunk, hist = codec.pack_blocks(x, 129, 3, 8, need_hist=True)
    assert len(chunk.seg_offsets) == 140_001 and int(hist.sum()) == x.numel()
    _round_trip(chunk, x)


def test_threads_have_reports_of_their_own(cuda_device):
    from adacode_b200 import codec
    xs = [synth.kv_tensor((1, 4, 128 * (3 + i), 64), seed=85 + i).to(cuda_device) for i in range(4)]
    want = [list(codec.pack_blocks(x, 129, 3, 128)[0].seg_offsets) for x in xs]
    errors = []

    def work(i):
        try:
            for _ in range(20):
                chunk, _ = codec.pack_blocks(xs[i], 129, 3, 128)
                assert list(chunk.seg_offsets) == want[i]
        except BaseException as e:          # noqa: BLE001 (handed to the test's thread)
            errors.append(e)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


class _Seen(TorchFunctionMode):
    def __init__(self):
        super().__init__()
        self.names = []

    def __torch_function__(self, func, types, args=(), kwargs=None):
        self.names.append(getattr(func, '__name__', str(func)))
        return func(*args, **(kwargs or {}))


class _Marked(torch.Tensor):
    seen = 0

    @classmethod
    def __torch_function__(cls, func, types, args=(), kwargs=None):
        cls.seen += getattr(func, '__name__', '') == 'copy_'
        return super().__torch_function__(func, types, args, kwargs or {})


def _cache(workspace='shared'):
    from adacode_b200 import Float11Cache
    return Float11Cache(StubConfig(1), 130, 3, block_size=128, layout='segmented_tiled', dense_workspace=workspace)


@pytest.mark.parametrize('workspace', ['shared', 'layer'])
def test_torch_functions_see_the_copies(cuda_device, workspace):
    """Modes and subclasses get the copies as calls of torch; the values are the same."""
    k, v = (synth.kv_tensor((1, 2, 303, 64), seed=s).to(cuda_device) for s in (1, 2))
    cache = _cache(workspace)
    cache.update(k[:, :, :300], v[:, :, :300], 0)
    new = k[:, :, 300:301], v[:, :, 300:301]
    with _Seen() as seen:
        dk, dv = cache.update(*new, 0)
    assert seen.names.count('copy_') >= 2
    assert torch.equal(dk, k[:, :, :301]) and torch.equal(dv, v[:, :, :301])
    _Marked.seen = 0
    dk, dv = cache.update(*(t[:, :, 301:302].as_subclass(_Marked) for t in (k, v)), 0)
    assert _Marked.seen >= 2
    assert torch.equal(dk.as_subclass(torch.Tensor), k[:, :, :302]) and torch.equal(dv.as_subclass(torch.Tensor), v[:, :, :302])


def test_tokens_of_other_types_and_devices(cuda_device):
    """copy_ converts, fetches and broadcasts; so does an append."""
    from adacode_b200.float_cache_utils import _Residual
    x = synth.kv_tensor((2, 2, 3, 64), seed=3)
    for states in (x.to(cuda_device).float(), x.to(cuda_device)[:1], x.to(cuda_device).transpose(1, 2).contiguous().transpose(1, 2)):
        r = _Residual()
        r.append(x.to(cuda_device), 128)
        r.append(states, 128)
        want = torch.cat([x.to(cuda_device), states.to(torch.bfloat16).expand(2, 2, 3, 64)], dim=2)
        assert r.length == 6 and torch.equal(r.tensor(), want)


def test_mixed_segments_are_refused(cuda_device):
    from adacode_b200 import codec
    cache = _cache()
    k = synth.kv_tensor((1, 2, 300, 64), seed=4).to(cuda_device)
    cache.update(k, k, 0)
    layer = cache.layers[0]
    layer._key_segments.append(codec.pack_blocks(k[:, :1, :128], 130, 3, 128)[0].segments()[0])
    with pytest.raises(ValueError, match='must share'):
        cache.materialize_layer(0)
