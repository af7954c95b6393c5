"""Fused attention's memory for partial results: calls on one stream share it, nobody else."""
import contextlib

import torch


def test_streams_and_captures_have_workspaces_of_their_own(monkeypatch):
    from adacode_b200 import _lib, attention, codec
    stream, capturing, spaces, sizes = [7], [False], [], []

    class Library:
        def adacode_decode_attn_workspace_bytes(self, B, Hq, D, n_splits):
            return B * Hq * n_splits * (D + 2) * 4

        def adacode_decode_attn(self, *args):
            spaces.append(args[-5])
            sizes.append(args[-4])
            return _lib.OK
    monkeypatch.setattr(attention._lib, 'lib', Library)
    scratch = codec._DeviceScratch(torch.device('cpu'))
    monkeypatch.setattr(attention, '_scratch_for', lambda device: scratch)
    monkeypatch.setattr(attention, 'on_device', lambda device: contextlib.nullcontext())
    monkeypatch.setattr(attention, 'stream_ptr', lambda device: stream[0])
    monkeypatch.setattr(torch.cuda, 'is_current_stream_capturing', lambda: capturing[0])

    def call(at, batch=1, captured=False):
        stream[0], capturing[0] = at, captured
        q, tail = torch.zeros(batch, 4, 64, dtype=torch.bfloat16), torch.zeros(batch, 2, 5, 64, dtype=torch.bfloat16)
        attention.decode_attention(q, [], [], tail, tail)
        assert sizes[-1] >= batch * 4 * 128 * 66 * 4
        return spaces[-1]
    first, second = call(7), call(8)
    assert first != second and call(7) == first and call(8) == second
    assert call(7, captured=True) != first and call(9, captured=True) and 9 not in scratch.partials.by_stream
    assert call(7, batch=64) and call(8) == second
