"""What of a model's weights is held when the cache is sized (engine/runner.py; host rules: no GPU)."""
import weakref

import pytest
import torch

from atom_b200.config import EngineConfig
from atom_b200.engine import runner as rn
from atom_b200.parts.recurrent import DecayedStateMixing


class _Sized(Exception):
    pass


def test_weights_that_a_part_has_stacked_are_given_back_before_the_cache_is_sized(tmp_path, monkeypatch):
    import tiny_nurinex

    tiny_nurinex.write_model(tiny_nurinex.CONFIGS["P"], str(tmp_path), 1)
    stacked, refs = tuple(f".{n}.weight" for n in "rkvg"), {}

    def load(model, path, dtype, device):
        tensors = load_weights(model, path, dtype, device)
        refs.update({k: weakref.ref(t) for k, t in tensors.items()})
        return tensors

    def after_load(self):      # the layers before have given theirs back: no more than one layer's are held twice
        gone_before.append(sum(k.endswith(stacked) and r() is None for k, r in refs.items()))
        after(self)

    def sized(self, needs):
        raise _Sized(self.weight_bytes, [k for k, r in refs.items() if k.endswith(stacked) and r() is not None])

    load_weights, gone_before, after = rn.load_weights, [], DecayedStateMixing.after_load
    monkeypatch.setattr(DecayedStateMixing, "after_load", after_load)
    monkeypatch.setattr(rn, "load_weights", load)
    monkeypatch.setattr(rn.ModelRunner, "_pages_from_free_memory", sized)
    monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
    monkeypatch.setattr(torch.cuda, "set_device", lambda device: None)
    monkeypatch.setattr(rn.native, "device_flags", lambda device: torch.zeros(2, dtype=torch.int32))
    monkeypatch.setattr(rn.native, "status_flag", lambda device: torch.zeros(1, dtype=torch.int32))
    with pytest.raises(_Sized) as e:
        rn.ModelRunner(EngineConfig(model=str(tmp_path), dtype="bfloat16"), device="cpu")
    weight_bytes, held = e.value.args
    assert sum(k.endswith(stacked) for k in refs) % 4 == 0 and any(k.endswith(stacked) for k in refs) and weight_bytes > 0
    assert not held, held
    assert len(gone_before) > 1 and gone_before == [4 * i for i in range(len(gone_before))]
