"""Handle.bind_current_stream on the host: how torch's current stream reaches the library."""
import pytest
import torch

from coral_b200 import blas


class FakeLib:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        return lambda *args: self.calls.append((name, *args)) or 0


def _handle():
    h = blas.Handle.__new__(blas.Handle)
    h.lib, h.h, h._raw, h._lasts = FakeLib(), None, None, True
    return h


class FakeStream:
    def __init__(self, stream_id, raw):
        self.stream_id, self.cuda_stream = stream_id, raw


@pytest.fixture
def fake_cuda(monkeypatch):
    now = {"stream": FakeStream(0, 0)}
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: now["stream"])
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda d: now["stream"].cuda_stream, raising=False)
    return now


def test_torchs_own_error_comes_first(monkeypatch):
    """CUDA is initialised by torch (which refuses in a forked child) before any raw handle is asked for."""
    def refuse():
        raise RuntimeError("Cannot re-initialize CUDA in forked subprocess")
    monkeypatch.setattr(torch.cuda, "_lazy_init", refuse)
    monkeypatch.setattr(torch._C, "_cuda_getDevice", lambda: 0, raising=False)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda d: 7, raising=False)
    h = _handle()
    with pytest.raises(RuntimeError, match="re-initialize"):
        h.bind_current_stream()
    assert h.lib.calls == []


def test_without_the_raw_getter(monkeypatch, fake_cuda):
    monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream")
    fake_cuda["stream"] = FakeStream(33, 0x7f0010)
    h = _handle()
    h.bind_current_stream()
    assert h.lib.calls[-1][2] == 0x7f0010


def test_only_external_streams_are_marked(fake_cuda):
    h = _handle()
    for stream, lasts in ((FakeStream(0, 0), True), (FakeStream(35, 0x7f0010), True),
                          (FakeStream(0x7f0020, 0x7f0020), False), (FakeStream(35, 0x7f0010), True)):
        fake_cuda["stream"] = stream
        h.lib.calls.clear()
        h.call("coral_saxpy", 1)
        names = [c[0] for c in h.lib.calls]
        assert h.lib.calls[0] == ("coral_bind_stream", None, stream.cuda_stream, lasts)
        assert names == ["coral_bind_stream", "coral_saxpy"] + ([] if lasts else ["coral_mark_stream"])
