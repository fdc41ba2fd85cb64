"""A second member on a stream of its own (parts/side_by_side.py): who waits for it (host rules: no GPU)."""
from types import SimpleNamespace

import pytest
import torch

from atom_b200.parts import side_by_side as sbs


class _Side:
    def __init__(self, log):
        self.log = log

    def run(self, work):
        self.log.append("fork")
        return work()

    def join(self):
        self.log.append("join")


@pytest.mark.parametrize("raises", [None, "first", "second", "meanwhile"])
def test_the_caller_waits_for_the_second_member_whatever_happens(raises, monkeypatch):
    """Both use the part's buffers, which the caller's next work takes over: it comes behind the second stream's also where a
    member raised."""
    monkeypatch.setattr(sbs.Beside, "may_run", staticmethod(lambda device: True))
    log = []

    def does(name):
        def work(*args):
            if raises == name:
                raise RuntimeError(name)
            log.append(name)
            return name
        return work

    part = object.__new__(sbs.SideBySide)
    part.members = {n: SimpleNamespace(forward=does(n)) for n in ("first", "second")}
    part._side = _Side(log)
    cache = SimpleNamespace(member=lambda name: None)
    go = lambda: part._members_forward(torch.zeros(sbs.OVERLAP_MIN_ROWS, 1), None, cache, True, does("meanwhile"))  # noqa: E731
    if raises is None:
        assert go() == (("first", "first"), ("second", "second"), "meanwhile")
        assert log == ["fork", "second", "meanwhile", "first", "join"]
    else:
        with pytest.raises(RuntimeError, match=raises):
            go()
        assert log[0] == "fork" and log[-1] == "join"
