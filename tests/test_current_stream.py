"""The current stream's handle comes from torch's public call where the raw one is missing."""


def test_public_call_without_the_raw_handle(monkeypatch):
    import torch

    from kete_b200 import _lib

    class Stream:
        cuda_stream = 1234

    monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: Stream)
    assert _lib._current_stream(0) == 1234


def test_raw_handle_when_there(monkeypatch):
    import torch

    from kete_b200 import _lib

    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda device: 40 + device,
                        raising=False)
    assert _lib._current_stream(2) == 42
