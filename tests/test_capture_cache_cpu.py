"""Row pointers made while a CUDA graph is being captured hold nothing before the graph's first replay (CPU: the capture is
a stand-in): a later call outside the graph must not find them in the cache."""
import torch

from cuequivariance_b200 import channelwise as cw


def test_nothing_made_under_capture_is_kept(monkeypatch):
    cache = cw._CsrCache()
    monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    idx, snd = torch.tensor([2, 0, 1, 1], dtype=torch.int64), torch.tensor([0, 1, 2, 0], dtype=torch.int64)
    captured = cache.get(idx, 3)
    cache.int32(snd)
    cache.get_passes(idx, snd, 3, 3, 2)
    assert cache.entries == []
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    eager = cache.get(idx, 3)
    assert eager[1] is not captured[1] and torch.equal(eager[1], torch.tensor([0, 1, 3, 4], dtype=torch.int32))
    assert cache.get(idx, 3)[1] is eager[1] and len(cache.entries) == 1
