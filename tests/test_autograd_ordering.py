"""The torch binding's stream ordering around a block: the block's own error is the one that is raised."""

import pytest

torch = pytest.importorskip("torch")

from cellflow_gb300 import autograd
from cellflow_gb300._lib import CellFlowError


class Lib:
    """Calls that succeed, but for the signal at the end."""

    def __init__(self, signal):
        self.signal, self.calls = signal, []

    def cf_stream_wait(self, handle, stream):
        self.calls.append("wait")
        return 0

    def cf_stream_signal(self, handle, stream):
        self.calls.append("signal")
        return self.signal


class World:
    handle = None


@pytest.fixture
def block(cflib, monkeypatch):
    def make(signal):
        lib = Lib(signal)
        monkeypatch.setattr(autograd, "load", lambda: lib)
        o = autograd._Ordered.__new__(autograd._Ordered)
        o.sim, o.stream = World(), 0
        return lib, o

    return make


def test_the_blocks_error_is_raised(block):
    lib, o = block(signal=2)
    with pytest.raises(ValueError, match="from the block"):
        with o:
            raise ValueError("from the block")
    assert lib.calls == ["wait", "signal"]  # (the caller's stream still waits for what was enqueued)


def test_a_failed_signal_is_raised_after_a_good_block(block):
    lib, o = block(signal=2)
    with pytest.raises(CellFlowError):
        with o:
            pass
    assert lib.calls == ["wait", "signal"]


def test_the_public_stream_call_is_enough(monkeypatch):
    monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: type("Stream", (), {"cuda_stream": 17})())
    assert autograd._current_stream() == 17
