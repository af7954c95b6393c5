"""Exponent histograms of values that do not lie in one window of fifteen exponents, and of runs of every length."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _count(x):
    return torch.bincount((x.contiguous().view(-1).view(torch.int16).int() >> 7) & 0xFF, minlength=256)


def _values(kind, shape, dev):
    g = torch.Generator(device=dev).manual_seed(len(kind))
    x = torch.randn(shape, generator=g, device=dev).to(torch.bfloat16)
    if kind == 'bits':
        x = torch.randint(-2 ** 15, 2 ** 15, shape, generator=g, device=dev).to(torch.int16).view(torch.bfloat16)
    elif kind == 'zeros':                                          # every other element
        x[..., ::2] = 0
    elif kind == 'outlier':                                        # a column far above all others sets every window
        x[..., 5] = 2.0 ** 60
    elif kind == 'first':                                          # only the first rows do
        x[:, :, :2] = 2.0 ** 60
    elif kind == 'halves':                                         # a change in the middle
        x[:, :, shape[2] // 2:] *= 2.0 ** -50
    elif kind == 'nan':
        x[torch.rand(shape, generator=g, device=dev) < 0.3] = float('nan')
    return x


@pytest.mark.parametrize('kind', ['normal', 'bits', 'zeros', 'outlier', 'first', 'halves', 'nan'])
def test_spread_of_exponents(cuda_device, kind):
    """Large enough that every warp counts several units and gives its windows up where it has to."""
    from adacode_b200 import codec
    x = _values(kind, (4, 8, 8192, 128), cuda_device)
    assert torch.equal(codec.exponent_hist(x).long(), _count(x))


@pytest.mark.parametrize('kind', ['normal', 'bits', 'outlier'])
@pytest.mark.parametrize('heads,D', [(1, 8), (1, 72), (1, 128), (2, 128), (3, 168), (4, 128), (5, 200)])
def test_heads_of_a_wider_projection(cuda_device, kind, heads, D):
    """Some heads of a [B, S, heads, D] projection: runs of heads * D elements, 1 to 125 vectors."""
    from adacode_b200 import codec
    x = _values(kind, (3, 3001, heads + 3, D), cuda_device).transpose(1, 2)[:, 2: 2 + heads]
    assert torch.equal(codec.exponent_hist(x).long(), _count(x))
