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


def test_weights_written_in_place_stay_where_captured_steps_read_them():
    """A program that writes new weights over a part's and has it look at them again: graphs captured before read the new ones."""
    from types import SimpleNamespace

    from atom_b200.parts import registry
    from atom_b200.parts.spec import PartSpec

    part = registry.build("mixer", PartSpec("decayed_state_mixing", {"hidden_size": 64, "num_heads": 4, "head_dim": 16, "decay_rank": 8,
                                                                     "norm_eps": 1e-5}))
    part.bind({n: torch.zeros(p.shape, dtype=torch.bfloat16) for n, p in part.params().items()},
              SimpleNamespace(dtype=torch.bfloat16, device=torch.device("cpu")))
    part.after_load()
    at, names = part._rkvg.data_ptr(), [f"w_{n}_weight" for n in "rkvg"]
    for i, n in enumerate(names):
        getattr(part, n).fill_(i + 1)
    part.after_load()
    assert part._rkvg.data_ptr() == at
    assert [float(m.float().mean()) for m in part._rkvg] == [1, 2, 3, 4]
    part.w_k_weight = torch.full((64, 64), 9.0, dtype=torch.bfloat16)      # (another tensor is taken up)
    part.after_load()
    assert [float(m.float().mean()) for m in part._rkvg] == [1, 9, 3, 4]
    assert [float(getattr(part, n).float().mean()) for n in names] == [1, 9, 3, 4]
