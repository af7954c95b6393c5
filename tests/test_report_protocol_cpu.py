"""The protocol of a report to the host, as far as it shows without a GPU: the host's side run against words written here, the
device's side read from its source."""
import ctypes
import os
import re

import numpy as np

from tests.conftest import ROOT


def _send_report() -> str:
    with open(os.path.join(ROOT, 'adacode_b200', 'csrc', 'adacode_pipeline.cuh')) as f:
        body = re.search(r'void send_report\(const Report &r\) \{\n(.*?)\n\}\n', f.read(), re.S)
    return body.group(1)


def test_word_and_token_are_one_scalar_store():
    """A vector store is several stores in no stated order: the host could see the token before the word."""
    stores = re.findall(r'"(st\.[^ ]+) ', _send_report())
    assert stores == ['st.relaxed.sys.global.b64'], stores


def test_the_host_takes_the_low_half_of_a_word_whose_high_half_is_the_token():
    from adacode_b200 import _lib
    words = np.array([7 << 32 | 0xFFFFFFFF, 7 << 32, 7 << 32 | 123456], dtype=np.uint64)
    out = np.zeros(3, dtype=np.uint32)
    assert _lib.lib().adacode_wait_report(words.ctypes.data_as(ctypes.c_void_p), 12, 7, out.ctypes.data_as(ctypes.c_void_p), None) == _lib.OK
    assert out.tolist() == [0xFFFFFFFF, 0, 123456]
