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


@pytest.mark.parametrize("design", DESIGNS)
@pytest.mark.parametrize("batch", [1, 8, 16])
def test_branches_of_a_wide_model(design, batch, monkeypatch):
    """Width 2,048, four layers, 300 tokens a sequence: products of hundreds of CTAs and attention by split keys beside a scan."""
    import bench
    from oracle_engine_b200.config.base import get_architecture
    from oracle_engine_b200.engine.batch import SequenceStep
    from oracle_engine_b200.engine.engine import Engine
    from oracle_engine_b200.parts import parallel
    raw = getattr(bench, design + "_shape")(2048, 4, 4096)
    config = get_architecture(raw["architecture"]).config_cls.from_dict(raw)

    def logits():
        eng = Engine.from_config(config, seed=3, dtype="bfloat16", max_tokens=16 * 384)
        slots = [eng.alloc() for _ in range(batch)]
        eng.step([SequenceStep(s, [(31 * b + 7 * j) % 4096 for j in range(300 - b)], []) for b, s in enumerate(slots)])
        return torch.stack([eng.step([SequenceStep(s, [(13 * i + b) % 4096], [0]) for b, s in enumerate(slots)]).clone() for i in range(5)])
    beside = logits()
    monkeypatch.setattr(parallel, "FORK_TOKENS", 0)
    after = logits()
    assert torch.isfinite(beside).all() and torch.equal(beside, after)


def test_only_in_a_capture():
    from oracle_engine_b200.engine.runtime import Runtime
    with pytest.raises(RuntimeError, match="captured"):
        Runtime(torch.bfloat16, torch.device("cuda:0")).fork(lambda: None, lambda: None)
