"""The current stream's handle, with and without torch's private call for it (no GPU)."""
from types import SimpleNamespace

from cuphoto import tsdf


def fake(private):
    t = SimpleNamespace(cuda=SimpleNamespace(current_device=lambda: 3,
                                             current_stream=lambda: SimpleNamespace(cuda_stream=77)),
                        _C=SimpleNamespace())
    if private:
        t._C._cuda_getCurrentRawStream = lambda device: 10 * device
    return t


def test_current_stream_handle(monkeypatch):
    monkeypatch.setattr(tsdf, "_torch", lambda: fake(True))
    assert tsdf._stream_handle(None) == 30
    monkeypatch.setattr(tsdf, "_torch", lambda: fake(False))
    assert tsdf._stream_handle(None) == 77
    assert tsdf._stream_handle(SimpleNamespace(cuda_stream=5)) == 5
