"""Who shares a pack scratch: packs on one stream, nobody else."""
import torch


def test_every_stream_has_a_scratch_of_its_own(monkeypatch):
    from adacode_b200 import codec
    scratch = codec._DeviceScratch.__new__(codec._DeviceScratch)
    monkeypatch.setattr(torch.cuda, 'Event', lambda: None)
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
    kept = [at(s) for s in range(100, 100 + codec._MAX_SCRATCH_STREAMS)]
    assert len(scratch.workspaces) == codec._MAX_SCRATCH_STREAMS
    assert all(at(100 + i) is ws for i, ws in enumerate(kept))
    assert at(12) is not second
