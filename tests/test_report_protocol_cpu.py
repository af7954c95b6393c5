"""The protocol of a report to the host, as far as it shows without a GPU: the host's side run against words written here, the
device's side read from its source."""
import ctypes
import os
import re

import numpy as np

from tests.conftest import ROOT


def _source(name: str) -> str:
    with open(os.path.join(ROOT, 'adacode_b200', 'csrc', name)) as f:
        return f.read()


def _send_report() -> str:
    return re.search(r'void send_report\(const Report &r\) \{\n(.*?)\n\}\n', _source('adacode_pipeline.cuh'), re.S).group(1)


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


def test_nothing_is_written_behind_a_report():
    """Whoever has the report may pack into the same scratch from another stream: the kernels send it last, and what they wrote
    is written for the whole GPU by then."""
    pipeline = _source('adacode_pipeline.cuh')
    end = pipeline[pipeline.index('if (pa.report.words != 0)'):]
    before, behind = end[:end.index('#endif')].split('send_report(pa.report)')
    assert 'acq_rel.gpu' in before and 'pa.done' not in behind
    tail = re.search(r'void __launch_bounds__\(kTailThreads\) k_flat_tail.*?\n\}\n', _source('adacode_kernels.cu'), re.S).group(0)
    assert tail.rstrip('}\n').endswith('send_report(a.report);')
    assert re.search(r'__threadfence\(\);[^\n]*\n\s*__syncthreads\(\);\n[^\n]*send_report', tail)
