"""The stream that operators launch on, with and without torch's raw-stream function."""
import importlib.util

import pytest
import torch

from socket_b200 import _lib


@pytest.mark.parametrize("raw", [True, False])
def test_current_stream_of_the_device(monkeypatch, raw):
    if raw:
        monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda index: 1000 + index, raising=False)
    else:
        monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)
    stream = lambda device=None: type("Stream", (), {"cuda_stream": 1000 + (3 if device is None or device.index is None else device.index)})
    monkeypatch.setattr(torch.cuda, "current_stream", stream)
    spec = importlib.util.spec_from_file_location("fresh_lib", _lib.__file__)
    fresh = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(fresh)
    assert fresh.stream_ptr() == fresh.stream_ptr(torch.device("cuda")) == 1003
    assert fresh.stream_ptr(torch.device("cuda", 1)) == 1001
