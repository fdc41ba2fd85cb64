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


def _part(log, does, width=2048):
    part = object.__new__(sbs.SideBySide)
    part.hidden_size = width
    part.members = {n: SimpleNamespace(forward=does(n)) for n in ("first", "second")}
    part._side = _Side(log)
    return part


@pytest.mark.parametrize("rows,width,forks", [(383, 2048, False), (384, 2048, True), (384, 1536, True), (512, 1024, False), (1279, 1024, False),
                                              (1280, 1024, True), (1024, 512, False), (2, 2048, False)])
def test_rows_from_which_the_second_member_has_its_own_stream(rows, width, forks, monkeypatch):
    monkeypatch.setattr(sbs.Beside, "may_run", staticmethod(lambda device: True))
    log = []
    _part(log, lambda name: lambda *args: name, width)._members_forward(torch.zeros(rows, 1), None, SimpleNamespace(member=lambda n: None), True)
    assert log == (["fork", "join"] if forks else [])


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

    part, cache = _part(log, does), SimpleNamespace(member=lambda name: None)
    go = lambda: part._members_forward(torch.zeros(sbs.OVERLAP_MIN_ROWS, 1), None, cache, True, does("meanwhile"))  # noqa: E731
    if raises is None:
        assert go() == (("first", "first"), ("second", "second"), "meanwhile")
        assert log == ["fork", "second", "meanwhile", "first", "join"]
    else:
        with pytest.raises(RuntimeError, match=raises):
            go()
        assert log[0] == "fork" and log[-1] == "join"
