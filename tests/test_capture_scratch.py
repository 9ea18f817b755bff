"""Whose scratch a call gets, without a GPU: allocation, initialisation and reuse per (device, stream, capture)."""
import pytest
import torch

from sol_execbench_b200_kernels_b200 import kernel


class _Recorder:
    """Stands in for the streams: `capture` is the capture that records them, 0 for none; `inits` what was initialised."""

    def __init__(self, monkeypatch):
        self.capture, self.inits, self.fail = 0, [], False
        monkeypatch.setattr(torch._C, "_cuda_isCurrentStreamCapturing", lambda: self.capture != 0)
        monkeypatch.setattr(kernel._cabi.lib, "gu_capture_id", lambda stream: self.capture, raising=False)
        self.kept = {}

    def init(self, ptr, nbytes, stream):
        self.inits.append((self.capture, ptr, nbytes, stream))
        return kernel._cabi.GU_ECUDA if self.fail else 0

    def take(self, stream=7, nbytes=4096, capture=0, device=0):
        self.capture = capture
        return kernel._workspace(torch.device("cpu", device), stream, nbytes, self.init, self.kept)


@pytest.fixture
def streams(monkeypatch):
    return _Recorder(monkeypatch)


def test_every_capture_has_scratch_of_its_own(streams):
    eager = streams.take()
    first, again = streams.take(capture=41), streams.take(capture=41)
    second = streams.take(capture=42)
    assert first is again
    assert len({t.data_ptr() for t in (eager, first, second)}) == 3
    # each one initialised once, by an operation of its own capture
    assert [(c, p) for c, p, _, _ in streams.inits] == [(0, eager.data_ptr()), (41, first.data_ptr()), (42, second.data_ptr())]
    assert streams.take() is eager and len(streams.inits) == 3


def test_a_stream_keeps_the_newest_capture_only(streams):
    eager = streams.take()
    for capture in range(1, 50):
        streams.take(capture=capture)
    assert len(streams.kept) == 2 and streams.take() is eager
    other = streams.take(stream=9, capture=49)  # a capture over two streams: one each
    assert len(streams.kept) == 3 and other is not streams.take(capture=49)


def test_scratch_grows_and_is_initialised_again(streams):
    for capture in (0, 5):
        small = streams.take(capture=capture)
        large = streams.take(nbytes=8192, capture=capture)
        assert large.numel() == 8192 and large is not small
        assert streams.take(capture=capture) is large
    assert [n for _, _, n, _ in streams.inits] == [4096, 8192] * 2


def test_a_failed_initialisation_is_not_kept(streams):
    streams.fail = True
    for capture in (0, 3):
        with pytest.raises(kernel._cabi.GateUpError):
            streams.take(capture=capture)
    assert not streams.kept
    streams.fail = False
    streams.take()
    assert len(streams.inits) == 3


def test_no_capture_without_a_device():
    assert kernel._cabi.lib.gu_capture_id(0) == 0
