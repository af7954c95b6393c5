"""What the copies of dense tokens inside a cache have to keep beside the bytes: tangents, recorded versions, refusals."""
import pytest
import torch
import torch.autograd.forward_ad as fwAD

from tests import synth
from tests.scenarios import StubConfig

pytestmark = pytest.mark.gpu


def _cache(workspace):
    from adacode_b200 import Float11Cache
    return Float11Cache(StubConfig(1), 130, 3, block_size=128, layout='segmented_tiled', dense_workspace=workspace)


def _dual(shape, dev, seed):
    g = torch.Generator('cpu').manual_seed(seed)
    x, t = (torch.randn(shape, generator=g).to(torch.bfloat16).to(dev) for _ in range(2))
    return fwAD.make_dual(x, t), t


def _check_tangents(dev, workspace, prompt):
    cache = _cache(workspace)
    k, v = (synth.kv_tensor((1, 2, prompt, 64), seed=s).to(dev) for s in (1, 2))
    cache.update(k, v, 0)
    with fwAD.dual_level():
        (kd, kt), (vd, vt) = _dual((1, 2, 3, 64), dev, 3), _dual((1, 2, 3, 64), dev, 4)
        for out, new, tangent in zip(cache.update(kd, vd, 0), (kd, vd), (kt, vt)):
            primal, got = fwAD.unpack_dual(out)
            assert torch.equal(primal[:, :, prompt:], fwAD.unpack_dual(new).primal)
            assert got is not None and torch.equal(got[:, :, prompt:], tangent) and not got[:, :, :prompt].any()


@pytest.mark.parametrize('workspace,prompt', [('shared', 60), ('layer', 60), ('layer', 300)])
def test_appended_tokens_keep_their_tangents(cuda_device, workspace, prompt):
    _check_tangents(cuda_device, workspace, prompt)


def test_dense_view_keeps_tangents(cuda_device):
    """Packed blocks have none; the tail behind them keeps its own."""
    _check_tangents(cuda_device, 'shared', 300)


def test_rows_under_transforms(cuda_device):
    """``torch.func`` wrappers are no plain rows: what ``copy_`` makes of them holds."""
    from adacode_b200.rows import copy_rows
    x, t = (torch.randn(2, 2, 3, 16, device=cuda_device).to(torch.bfloat16) for _ in range(2))

    def copied(a):
        out = torch.empty_like(a)
        copy_rows([(a, out)])
        return out

    out, tangent = torch.func.jvp(copied, (x,), (t,))
    assert torch.equal(out, x) and torch.equal(tangent, t)
    assert torch.equal(torch.func.vmap(copied)(x[None].expand(3, 2, 2, 3, 16)), x[None].expand(3, 2, 2, 3, 16))


def test_overwritten_workspace_is_noticed(cuda_device):
    """Dense keys saved for a backward pass and overwritten by the next call: autograd refuses."""
    cache = _cache('shared')
    k, v = (synth.kv_tensor((1, 2, 303, 64), seed=s).to(cuda_device) for s in (1, 2))
    cache.update(k[:, :, :300], v[:, :, :300], 0)
    dense, _ = cache.update(k[:, :, 300:301], v[:, :, 300:301], 0)
    q = torch.ones(1, 2, 1, 64, dtype=torch.bfloat16, device=cuda_device, requires_grad=True)
    scores = q @ dense.transpose(2, 3)
    cache.update(k[:, :, 301:302], v[:, :, 301:302], 0)
    with pytest.raises(RuntimeError, match='modified by an inplace operation'):
        scores.float().sum().backward()


def test_what_copy_refuses_is_refused(cuda_device):
    from adacode_b200 import codec
    from adacode_b200.rows import copy_rows
    x = torch.randn(2, 2, 3, 16, device=cuda_device).to(torch.bfloat16)
    with torch.inference_mode():
        frozen = torch.zeros_like(x)
    with pytest.raises(RuntimeError, match='InferenceMode'):
        copy_rows([(x, frozen)])
    with pytest.raises(RuntimeError, match='single memory location'):
        copy_rows([(x, torch.zeros(2, 1, 3, 16, dtype=torch.bfloat16, device=cuda_device).expand(2, 2, 3, 16))])
    k = synth.kv_tensor((1, 2, 140, 64), seed=1).to(cuda_device)
    segs = codec.pack_blocks(k[:, :, :128], 130, 3, 128)[0].segments()
    with torch.inference_mode():
        dense = torch.zeros_like(k)
    with pytest.raises(RuntimeError, match='InferenceMode'):
        codec.unpack_with_tails([(segs, None, dense, k[:, :, 128:].contiguous())], 128, 12)


@pytest.mark.parametrize('nk,nv', [(1, 2), (3, 2)])
def test_uneven_tails_are_refused(cuda_device, nk, nv):
    """Keys and values of different numbers of tokens: no dense view with rows that nobody wrote."""
    cache = _cache('shared')
    k, v = (synth.kv_tensor((1, 2, 303, 64), seed=s).to(cuda_device) for s in (1, 2))
    cache.update(k[:, :, :300], v[:, :, :300], 0)
    with pytest.raises(RuntimeError):
        cache.update(k[:, :, 300: 300 + nk], v[:, :, 300: 300 + nv], 0)


def test_dense_too_small_for_its_parts(cuda_device):
    from adacode_b200 import codec
    k = synth.kv_tensor((1, 2, 300, 64), seed=1).to(cuda_device)
    segs = codec.pack_blocks(k[:, :, :256], 130, 3, 128)[0].segments()
    tail = k[:, :, 256:].contiguous()
    for prefix, rows, length in ((256, 44, 299), (200, 44, 300), (300, 0, 299)):
        dense = torch.zeros(1, 2, length, 64, dtype=torch.bfloat16, device=cuda_device)
        with pytest.raises(ValueError, match='do not fit'):
            codec.unpack_with_tails([(segs, None, dense, tail)], prefix, rows)
        assert not dense.any()


@pytest.mark.parametrize('H,D,rows', [(1, 128, 5000), (2, 64, 40001), (1, 2048, 700), (3, 72, 3000)])
def test_tails_longer_than_the_packed_part(cuda_device, H, D, rows):
    """One packed block: the rows decide the launch's grid, most CTAs have no tile.  2048: the wide geometry, 72: the
    direct kernels."""
    from adacode_b200 import codec
    g = torch.Generator(device=cuda_device).manual_seed(rows)
    x = [torch.randn(1, H, 128 + rows, D, generator=g, device=cuda_device).to(torch.bfloat16) for _ in range(2)]
    parts = [(codec.pack_blocks(t[:, :, :128], 129, 3, 128)[0].segments(), None, torch.zeros_like(t), t[:, :, 128:]) for t in x]
    codec.unpack_with_tails(parts, 128, rows)
    for t, (_, _, dense, _) in zip(x, parts):
        assert torch.equal(dense.view(torch.int16), t.view(torch.int16))
    codec.check_device_status(cuda_device)


@pytest.mark.parametrize('workspace,prompt', [('shared', 60), ('shared', 300), ('layer', 300)])
def test_gradients_of_appended_tokens(cuda_device, workspace, prompt):
    cache = _cache(workspace)
    k, v = (synth.kv_tensor((2, 2, prompt, 64), seed=s).to(cuda_device) for s in (1, 2))
    cache.update(k, v, 0)
    kn, vn = (synth.kv_tensor((2, 2, 3, 64), seed=s).to(cuda_device).requires_grad_() for s in (3, 4))
    dk, dv = cache.update(kn, vn, 0)
    assert torch.equal(dk[:, :, prompt:], kn) and torch.equal(dv[:, :, :prompt], v)
    w = torch.randn(2, 2, prompt + 3, 64, device=cuda_device)
    ((dk.float() + 2 * dv.float()) * w).sum().backward()
    want = w[:, :, prompt:].to(torch.bfloat16)
    assert torch.equal(kn.grad, want) and torch.equal(vn.grad, 2 * want)
    from adacode_b200.float_cache_utils import _GLOBAL_WORKSPACE
    _GLOBAL_WORKSPACE.release()               # (it took part in this graph)
