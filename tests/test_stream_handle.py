"""The binding's handle of the current stream, with and without torch's private function."""
import types

import pytest
import torch

from conftest import load_pkg


@pytest.mark.parametrize("private", [True, False])
def test_current_stream(monkeypatch, private):
    binding = load_pkg().binding
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: types.SimpleNamespace(cuda_stream=77))
    if private:
        monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda d: 1000 + d, raising=False)
    else:
        monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
    assert binding.stream_handle() == (1003 if private else 77)
    assert binding.stream_handle(5) == 5
    assert binding.stream_handle(types.SimpleNamespace(cuda_stream=9)) == 9
