"""The host's side of a step's arrays (engine/batch.py): how long what the device reads stays as it is, and when it is there."""
from types import SimpleNamespace

import pytest
import torch

from atom_b200.cache import CacheManager
from atom_b200.engine import batch


class _Event:
    def __init__(self, log):
        self.log = log

    def synchronize(self):
        self.log.append(self)


def test_buffers_are_given_back_when_the_device_has_read_them():
    log = []
    ring = batch._HostRing(4)
    ring.events[1], ring.events[3] = one, two = _Event(log), _Event(log)
    del ring
    assert log == [one, two]


@pytest.mark.parametrize("mixed", [False, True])
def test_a_step_that_is_not_replayed_finds_its_arrays_complete(mixed, monkeypatch):
    """A kernel fills the fixed arrays, and a step's kernels may read them before they wait for the launch in front: only a graph,
    which waits for all of it, may be launched straight behind."""
    log = []
    host = torch.zeros(4096, dtype=torch.int32)
    stream = SimpleNamespace(synchronize=lambda: log.append("wait"))
    monkeypatch.setattr(batch, "_HostRing", lambda: SimpleNamespace(acquire=lambda n: (0, host, host.numpy()), sent=lambda k: None))
    monkeypatch.setattr(batch.native, "step_arrays", lambda *a: log.append("arrays"))
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: stream)
    builder = batch.StepBuilder(CacheManager({}, 16, 4, 4), "cpu", 100, torch.zeros(1, dtype=torch.int32))
    build = (lambda **kw: builder.build_fixed_mixed([], [], 32, 4, 8, **kw)) if mixed else (lambda **kw: builder.build_fixed([], [], 4, 8, **kw))
    build()
    assert log == ["arrays", "wait"]
    build(replayed=True)
    assert log == ["arrays", "wait", "arrays"]
