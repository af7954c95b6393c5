"""Flat packs of views that begin anywhere: the kernels get 16-byte boundaries."""
import pytest
import torch


@pytest.mark.parametrize('per_call', [1 << 30, 2048])
@pytest.mark.parametrize('n', [96, 1024, 1040, 2048, 4096 + 1032])
def test_the_kernels_see_aligned_tensors(monkeypatch, n, per_call):
    from adacode_b200 import _lib, codec, compress_bitmap_merge
    seen = []

    class Native:
        @staticmethod
        def pack_flat(x, right, nbits, block, cap, hist, ws):
            seen.append(x)
            assert x.data_ptr() % 16 == 0
            m = x.numel()
            return (torch.zeros(m, dtype=torch.uint8), torch.zeros(m * nbits // 8, dtype=torch.uint8), torch.zeros(cap, dtype=torch.uint8),
                    torch.zeros(-(-m // block), dtype=torch.int32), 0, 0)
    monkeypatch.setattr(_lib, 'native', lambda: Native)
    monkeypatch.setattr(codec, '_scratch_for', lambda device: codec._DeviceScratch(torch.device('cpu')))
    monkeypatch.setattr(codec, 'stream_ptr', lambda device: 0)
    monkeypatch.setattr(compress_bitmap_merge, '_MAX_ELEMS_PER_CALL', per_call)
    room = torch.arange(n + 5, dtype=torch.int16).view(torch.bfloat16)
    view = room[5:]
    assert view.data_ptr() % 16
    compress_bitmap_merge.CompressorBitMap(129, 3).compress(view)
    assert torch.equal(torch.cat(seen).view(torch.int16), view.view(torch.int16))
