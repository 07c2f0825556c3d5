"""The stream that a call runs on, without a GPU: torch's raw handle, the public
call where torch does not have it, and no stream before CUDA is initialised."""
import pytest

torch = pytest.importorskip("torch")


def test_stream_of(monkeypatch):
    from plenvdb_gb300 import _lib as L

    class Stream:
        cuda_stream = 4321

    monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
    monkeypatch.setattr(torch.cuda, "is_initialized", lambda: False)
    assert L.stream_of() is None
    monkeypatch.setattr(torch.cuda, "is_initialized", lambda: True)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: Stream)
    monkeypatch.setattr(torch._C, "_cuda_getDevice", lambda: 3, raising=False)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda d: 1000 + d, raising=False)
    assert L.stream_of() == 1003
    monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream")
    assert L.stream_of() == 4321
    monkeypatch.delattr(torch._C, "_cuda_getDevice")
    assert L.stream_of() == 4321
