"""The row-copy kernel against ``Tensor.copy_``, alone and along with an unpack launch; what it leaves to ``copy_``."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _views(dev, B, H, T, D, seed):
    g = torch.Generator('cpu').manual_seed(seed)
    x = torch.randn(B, H, T, D, generator=g).to(torch.bfloat16).to(dev)
    longer = torch.zeros(B, H, T + 5, D, dtype=torch.bfloat16, device=dev)
    longer[:, :, 2:2 + T] = x
    odd = torch.zeros(B, H, T, D + 1, dtype=torch.bfloat16, device=dev)
    odd[..., 1:] = x
    # contiguous, a slice of a buffer, a projection, one head for all, rows on 2-byte boundaries (left to copy_)
    return [x, longer[:, :, 2:2 + T], x.transpose(1, 2).contiguous().transpose(1, 2), x[:, :1].expand(B, H, T, D), odd[..., 1:]]


@pytest.mark.parametrize('B,H,T,D', [(1, 1, 1, 8), (2, 3, 1, 128), (3, 8, 77, 80), (1, 2, 300, 64), (2, 1, 5, 20)])
def test_copies_equal_copy_(cuda_device, B, H, T, D):
    from adacode_b200.rows import copy_rows
    for a in _views(cuda_device, B, H, T, D, 1):
        for b in _views(cuda_device, B, H, T, D, 2)[:3]:
            out = [torch.full((B, H, T + 9, D), 7.0, dtype=torch.bfloat16, device=cuda_device) for _ in range(2)]
            copy_rows([(a, out[0][:, :, 4:4 + T]), (b, out[1][:, :, 9:])])
            for o, src, lo in zip(out, (a, b), (4, 9)):
                want = torch.full_like(o, 7.0)
                want[:, :, lo:lo + T].copy_(src)
                assert torch.equal(o, want)


def test_what_copy_does_beyond_rows_still_works(cuda_device):
    from adacode_b200.rows import copy_rows
    dst = torch.zeros(2, 2, 3, 16, dtype=torch.bfloat16, device=cuda_device)
    copy_rows([(torch.ones(2, 2, 3, 16), dst)])                             # another device and type
    assert bool((dst == 1).all())
    copy_rows([(torch.full((1, 2, 3, 16), 2.0, dtype=torch.bfloat16, device=cuda_device), dst)])       # broadcast
    assert bool((dst == 2).all())
    src = torch.randn(2, 2, 3, 16, device=cuda_device).to(torch.bfloat16).requires_grad_()
    out = torch.zeros(2, 2, 3, 16, dtype=torch.bfloat16, device=cuda_device)
    copy_rows([(src, out)])                                                 # the gradient is recorded
    out.float().sum().backward()
    assert bool((src.grad == 1).all())
    with pytest.raises(RuntimeError):
        copy_rows([(torch.zeros(2, 2, 4, 16, dtype=torch.bfloat16, device=cuda_device), dst)])


@pytest.mark.parametrize('D', [72, 128])
@pytest.mark.parametrize('rows', [0, 1, 127, 300])
def test_unpack_with_tails(cuda_device, D, rows):
    """72: the direct kernels, with the rows in a launch of their own."""
    from adacode_b200 import codec
    g = torch.Generator('cpu').manual_seed(rows + D)
    x = [torch.randn(2, 3, 256 + rows, D, generator=g).to(torch.bfloat16).to(cuda_device) for _ in range(2)]
    parts = []
    for t in x:
        segs = codec.pack_blocks(t[:, :, :256], 129, 3, 128)[0].segments()
        tail = torch.zeros(2, 3, max(rows, 1) + 11, D, dtype=torch.bfloat16, device=cuda_device)
        tail[:, :, :rows] = t[:, :, 256:]
        parts.append((segs, codec.build_segment_table(segs), torch.zeros_like(t), tail))
    codec.unpack_with_tails(parts, 256, rows)
    for t, (_, _, dense, _) in zip(x, parts):
        assert torch.equal(dense.view(torch.int16), t.view(torch.int16))
    codec.check_device_status(cuda_device)
