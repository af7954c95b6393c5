"""The adjuster's choice on the device for histograms with ties, empty and full bins, and counts as large as they get."""
import numpy as np
import pytest
import torch

from oracle import float11_oracle as O

pytestmark = pytest.mark.gpu


def test_choices(cuda_device):
    from adacode_b200 import codec
    rng = np.random.default_rng(5)
    hists = [rng.integers(0, 1000, 256) for _ in range(20)]
    hists += [np.ones(256, np.int64), np.zeros(256, np.int64), rng.integers(0, 3, 256), np.eye(256, dtype=np.int64)[0], np.eye(256, dtype=np.int64)[255]]
    big = np.zeros(256, np.int64)
    big[[3, 3 + 32, 200]] = 2 ** 31 - 1, 2 ** 31 - 1, 2 ** 31 - 2
    hists += [big, np.where(np.arange(256) % 17 == 0, 2 ** 30, 5)]
    for width in (2, 3, 7, 8, 15, 16, 40):
        h = np.zeros(256, np.int64)
        h[100: 100 + width] = rng.integers(1, 50, width) * 1000
        hists.append(h)
    got = codec.choose_params_device(torch.tensor(np.stack(hists), dtype=torch.int32, device=cuda_device)).cpu().tolist()
    for h, (right, nbits) in zip(hists, got):
        try:
            want = tuple(O.choose_params(np.asarray(h, np.int64)))
        except IndexError:
            assert nbits == 0
            continue
        if want[1] == 0:
            assert nbits == 0
        else:
            assert (right, nbits) == want
