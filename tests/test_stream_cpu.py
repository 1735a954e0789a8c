"""The stream that the wrappers hand to the C API, with and without torch's inner shortcut."""
import types

import torch

from ccbench_b200 import comm


def test_stream_pointer_by_either_way(monkeypatch):
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)
    monkeypatch.setattr(comm, "_raw_stream", lambda device: 0x1000 + device)
    assert comm.current_stream_ptr().value == 0x1003
    monkeypatch.setattr(comm, "_raw_stream", None)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: types.SimpleNamespace(cuda_stream=0x2000))
    assert comm.current_stream_ptr().value == 0x2000
    assert comm.Communicator._stream().value == 0x2000
