"""The host's side of a step's arrays (engine/batch.py): how long what the device reads stays as it is."""
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
