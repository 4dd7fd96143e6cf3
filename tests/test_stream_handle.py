"""The current stream's handle where torch lacks the internal call that the
wrappers prefer: the public one gives it."""
from types import SimpleNamespace

import torch

from atag import lib


def test_handle_without_the_internal_call(monkeypatch):
    monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: SimpleNamespace(cuda_stream=77))
    assert lib.current_stream() == 77


def test_handle_by_the_internal_call(monkeypatch):
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda device: 100 + device, raising=False)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)
    assert lib.current_stream() == 103
