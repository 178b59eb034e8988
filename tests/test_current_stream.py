"""The Python binding's current stream (rfx._stream_ptr) with and without torch's raw binding."""
from __future__ import annotations

import types

import pytest
import torch

import rfx


@pytest.mark.parametrize("private", [True, False])
def test_handle_of_the_current_device(monkeypatch, private: bool) -> None:
    monkeypatch.setattr(rfx, "_raw_stream", None)
    monkeypatch.setattr(rfx, "_current_device", None)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)
    if private:
        monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda device: 100 + device,
                            raising=False)
    else:
        monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
        monkeypatch.setattr(torch.cuda, "current_stream",
                            lambda device=None: types.SimpleNamespace(cuda_stream=100 + device))
    assert rfx._stream_ptr(None) == 103
    assert rfx._stream_ptr(None) == 103
    assert rfx._stream_ptr(7) == 7


@pytest.mark.gpu
def test_follows_the_current_stream() -> None:
    for stream in (torch.cuda.default_stream(), torch.cuda.Stream()):
        with torch.cuda.stream(stream):
            assert rfx._stream_ptr(None) == stream.cuda_stream
