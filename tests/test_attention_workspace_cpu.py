"""Fused attention's partial results: two calls that are under way at a time do not share the memory for them."""
import contextlib
import threading

import torch


def test_calls_of_two_threads_have_workspaces_of_their_own(monkeypatch):
    from adacode_b200 import _lib, attention
    both, spaces = threading.Barrier(2), []

    class Library:
        def adacode_decode_attn_workspace_bytes(self, B, Hq, D, n_splits):
            return B * Hq * n_splits * (D + 2) * 4

        def adacode_decode_attn(self, *args):
            spaces.append(args[-5])
            both.wait(10)
            return _lib.OK
    monkeypatch.setattr(attention._lib, 'lib', Library)
    monkeypatch.setattr(attention, '_scratch_for', lambda device: type('Scratch', (), {'status': torch.zeros(2, dtype=torch.int32)}))
    monkeypatch.setattr(attention, 'on_device', lambda device: contextlib.nullcontext())
    monkeypatch.setattr(attention, 'stream_ptr', lambda device: 0)
    q, tail = torch.zeros(1, 4, 64, dtype=torch.bfloat16), torch.zeros(1, 2, 5, 64, dtype=torch.bfloat16)
    threads = [threading.Thread(target=attention.decode_attention, args=(q, [], [], tail, tail)) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(spaces) == 2 and spaces[0] != spaces[1]
