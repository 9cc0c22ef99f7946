"""The current stream's handle with and without torch's direct query of it."""

import importlib

import torch

from latticeboltzmann_gb300 import _tensor


class Stream:
    def __init__(self, device):
        self.cuda_stream = ("stream of", device)


class OnDevice:
    device = torch.device("cuda", 3)

    def get_device(self):
        return 3


def test_with_and_without_the_direct_query(monkeypatch):
    monkeypatch.setattr(torch.cuda, "current_stream", Stream)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 5)
    try:
        monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda index: ("raw", index), raising=False)
        importlib.reload(_tensor)
        assert _tensor.stream_of(torch.device("cuda", 2)) == ("raw", 2)
        assert _tensor.stream_of(torch.device("cuda")) == ("raw", 5)
        assert _tensor.stream_handle(OnDevice()) == ("raw", 3)
        monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream")
        importlib.reload(_tensor)
        assert _tensor.stream_of(torch.device("cuda", 2)) == ("stream of", 2)
        assert _tensor.stream_of(torch.device("cuda")) == ("stream of", 5)
        assert _tensor.stream_handle(OnDevice()) == ("stream of", 3)
    finally:
        monkeypatch.undo()
        importlib.reload(_tensor)
