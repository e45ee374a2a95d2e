"""Which calls share a workspace: those of one thread on one stream, which are ordered, and no others."""
from __future__ import annotations

import threading

import pytest
import torch

from cupynumeric_b200 import _lib
from cupynumeric_b200.runtime import Runtime


class Fake(Runtime):
    """Streams are numbers and device memory is the host's."""

    def __init__(self, monkeypatch):
        super().__init__()
        self.stream, self.dev, self.full_at = 1, 0, None
        monkeypatch.setattr(torch.cuda, "current_device", lambda: self.dev)
        monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
        monkeypatch.setattr(torch.cuda, "synchronize", lambda dev=None: None)

    @property
    def device(self):
        return torch.device("cpu")

    def stream_handle(self):
        return self.stream

    def _bytes(self, nbytes):
        if self.full_at is not None and sum(s.nbytes for s in self._kept.values()) + nbytes > self.full_at:
            raise torch.cuda.OutOfMemoryError("no room")
        raw = torch.zeros(nbytes + 256, dtype=torch.uint8)
        at = -raw.data_ptr() % 256
        return raw[at : at + nbytes]


@pytest.fixture
def run(monkeypatch):
    return Fake(monkeypatch)


def _in_thread(f):
    got = []
    t = threading.Thread(target=lambda: got.append(f()))
    t.start()
    t.join()
    return got[0]


def test_streams_threads_and_devices_do_not_share(run):
    first = run.workspace(1000)
    assert run.workspace(2000) is first            # (the smallest is larger)
    run.stream = 2
    second = run.workspace(1000)
    third = _in_thread(lambda: run.workspace(1000))
    run.dev = 1
    fourth = run.workspace(1000)
    assert len({w.data_ptr() for w in (first, second, third, fourth)}) == 4
    run.stream, run.dev = 1, 0
    assert run.workspace(1000) is first
    larger = run.workspace(1 << 17)
    assert larger.numel() >= 1 << 17 and run.workspace(1000) is larger


def test_what_is_kept_is_bounded_and_given_back(run):
    ws = {}
    for run.stream in range(Runtime.KEPT + 3):
        ws[run.stream] = run.workspace(1000)
    assert len(run._kept) == Runtime.KEPT
    run.stream = 0
    assert run.workspace(1000) is not ws[0]        # (it went first)
    run.stream = Runtime.KEPT + 2
    assert run.workspace(1000) is ws[run.stream]
    run.full_at = 1 << 20
    assert run.workspace(1 << 20).numel() == 1 << 20 and len(run._kept) == 1   # room is made of what the others keep
    run.release_workspace()
    assert not run._kept
    with pytest.raises(torch.cuda.OutOfMemoryError):
        run.workspace((1 << 20) + 1)


def test_what_the_others_hold_is_bounded_too(run, monkeypatch):
    monkeypatch.setattr(Runtime, "KEPT_BYTES", 3 << 20)
    for run.stream in range(4):
        run.workspace(2 << 20)
    assert sorted(k[1] for k in run._kept) == [2, 3]


@pytest.mark.parametrize("streams", [2, 66])
def test_a_failure_on_any_stream_is_raised_once(run, streams):
    for run.stream in range(streams):
        own = run.scratch(1000, run.dev, run.stream)
        own.status.fill_(5 if run.stream == 1 else 0)
        run.note_sort(own)
    assert len(run._sticky) <= Runtime.STICKY < 66
    with pytest.raises(_lib.B2SError):
        run.raise_pending()
    run.raise_pending()
