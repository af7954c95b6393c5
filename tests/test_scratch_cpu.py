"""Who shares a pack scratch (packs on one stream, nobody else) and the bytes that results are read back into (one thread)."""
import contextlib
import ctypes
import threading

import numpy as np
import torch


def test_every_stream_has_a_scratch_of_its_own(monkeypatch):
    from adacode_b200 import codec
    scratch = codec._DeviceScratch.__new__(codec._DeviceScratch)
    scratch.__init__(torch.device('cpu'))
    now = [0]
    monkeypatch.setattr(codec, 'stream_ptr', lambda device: now[0])

    def at(stream, n_tiles=4):
        now[0] = stream
        return scratch.workspace_for(n_tiles, 128 * 128)
    first, second = at(11), at(12)
    assert first.data_ptr() != second.data_ptr()
    assert at(11) is first and at(12) is second and not first.any()
    grown = at(11, 400)
    assert grown.numel() > first.numel() and at(11) is grown and at(12) is second
    # what streams keep is bounded, and the newest stay
    kept = [at(s) for s in range(100, 100 + codec._MAX_STREAMS)]
    assert len(scratch.packs.by_stream) == codec._MAX_STREAMS
    assert all(at(100 + i) is ws for i, ws in enumerate(kept))
    assert at(12) is not second


def test_threads_read_back_into_bytes_of_their_own(monkeypatch):
    """Two threads whose copies are both under way before either takes its result."""
    from adacode_b200 import _lib, codec
    both = threading.Barrier(2)

    class Library:
        def adacode_copy_to_host(self, src, dst, nbytes, stream):
            ctypes.memmove(dst, src, nbytes)
            return _lib.OK

    class Event:
        def record(self, stream):
            pass

        def synchronize(self):
            both.wait(10)
    monkeypatch.setattr(codec._lib, 'lib', Library)
    monkeypatch.setattr(torch.cuda, 'Event', Event)
    monkeypatch.setattr(torch.cuda, 'current_stream', lambda device: type('Stream', (), {'cuda_stream': 0}))
    monkeypatch.setattr(torch.Tensor, 'pin_memory', lambda self: self)
    monkeypatch.setattr(codec, 'on_device', lambda device: contextlib.nullcontext())
    scratch = type('Scratch', (), {'mailbox': None, 'mail_event': Event()})()
    monkeypatch.setattr(codec, '_scratch_for', lambda device: scratch)
    if hasattr(codec, '_Mailbox'):
        monkeypatch.setattr(codec, '_mailbox', codec._Mailbox())
    sent = [torch.full((256,), 5 + i, dtype=torch.int32) for i in range(2)]
    got = [None, None]

    def work(i):
        got[i] = codec.read_back(sent[i])
    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(np.array_equal(got[i], sent[i].numpy()) for i in range(2)), got
