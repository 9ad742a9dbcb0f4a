"""Two mixers of a layer as two branches of a captured decode step: the bits of the step that runs them one after the other."""
import pytest
import torch

import fovirax_models
import fuvipel_models
import mavinex_models

pytestmark = pytest.mark.gpu
DESIGNS = {"fovirax": fovirax_models, "fuvipel": fuvipel_models, "mavinex": mavinex_models}


def _logits(folder, dtype, batch):
    from oracle_engine_b200.engine.batch import SequenceStep
    from oracle_engine_b200.engine.engine import Engine
    eng = Engine.from_pretrained(folder, dtype=dtype, max_tokens=17 * 128)
    slots = [eng.alloc() for _ in range(batch)]
    out = []
    for i in range(6):
        n = 1 if i else 3
        steps = [SequenceStep(s, [(17 * b + 5 * i + j) % 90 for j in range(n if i else n + b)], [n - 1]) for b, s in enumerate(slots)]
        out.append(eng.step(steps).clone())
    return torch.stack(out), eng


@pytest.mark.parametrize("design", DESIGNS)
@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("batch", [1, 5, 16, 17])
def test_branches_beside_each_other(design, dtype, batch, tmp_path, monkeypatch):
    from oracle_engine_b200.engine.runtime import Runtime
    from oracle_engine_b200.parts import parallel
    folder = DESIGNS[design].write(tmp_path, DESIGNS[design].REAL, 11)
    forks, fork = [], Runtime.fork

    def counted(self, first, second):
        forks.append(1)
        fork(self, first, second)
    monkeypatch.setattr(Runtime, "fork", counted)
    beside, eng = _logits(folder, dtype, batch)
    assert bool(forks) == (batch <= parallel.FORK_TOKENS)
    monkeypatch.setattr(parallel, "FORK_TOKENS", 0)
    after, _ = _logits(folder, dtype, batch)
    assert torch.isfinite(beside).all() and torch.equal(beside, after)


def test_only_in_a_capture():
    from oracle_engine_b200.engine.runtime import Runtime
    with pytest.raises(RuntimeError, match="captured"):
        Runtime(torch.bfloat16, torch.device("cuda:0")).fork(lambda: None, lambda: None)
