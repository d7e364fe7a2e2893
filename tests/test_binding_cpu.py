"""The Python binding's current stream with and without torch's raw-handle calls (not public API)."""
import types

import pytest
import torch

import ckks_b200 as cb


@pytest.mark.parametrize("raw", [True, False])
def test_current_stream(monkeypatch, raw):
    monkeypatch.setattr(cb, "_raw_stream", None)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: types.SimpleNamespace(cuda_stream=11))
    if raw:
        monkeypatch.setattr(torch._C, "_cuda_getDevice", lambda: 3, raising=False)
        monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda device: 100 + device, raising=False)
    else:
        monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
    assert cb._stream(None) == (103 if raw else 11)
    assert cb._stream(0) == 0 and cb._stream(7) == 7
