"""A captured step's recurrent layers take the scan that its sequences' real lengths ask for, not its padded size's."""
import pytest
import torch

import fuvipel_models

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def folder(tmp_path_factory):
    return fuvipel_models.write(tmp_path_factory.mktemp("scan"), fuvipel_models.REAL, 11)


def _step(eng, lens, seed):
    from oracle_engine_b200.engine.batch import SequenceStep
    g = torch.Generator().manual_seed(seed)
    slots = [eng.alloc() for _ in lens]
    out = eng.step([SequenceStep(s, torch.randint(0, 1000, (n,), generator=g).tolist(), [n - 1]) for s, n in zip(slots, lens)]).clone()
    for s in slots:
        eng.free(s)
    return out


def test_the_scan_of_a_captured_step(folder, monkeypatch):
    from oracle_engine_b200.csrc import ops
    from oracle_engine_b200.engine.engine import Engine
    calls = []
    for name in ("delta_chunks", "delta_rule_scan", "decay_chunks", "decay_scan"):
        monkeypatch.setattr(ops, name, lambda *a, name=name, fn=getattr(ops, name): (calls.append(name), fn(*a)))
    graphs = Engine.from_pretrained(folder, dtype="bfloat16", max_tokens=64 * 128)
    plain = Engine.from_pretrained(folder, dtype="bfloat16", max_tokens=64 * 128, use_graphs=False)
    walk, chunks = ["decay_scan", "delta_rule_scan", "decay_scan"], ["decay_chunks", "delta_chunks", "decay_chunks"]
    # 256 padded tokens of 32 padded sequences twice, of 4 twice, of 1; then 64 of 8
    steps = [([7] * 32, walk), ([200] + [1] * 30, ["decay_chunks", "delta_rule_scan", "decay_chunks"]), ([50] * 4, walk), ([200, 3, 2], chunks),
             ([250], chunks), ([5] * 8, walk)]
    for turn in range(4):                                     # run directly, captured, replayed twice
        for i, (lens, want) in enumerate(steps):
            calls.clear()
            got = _step(graphs, lens, 10 * i + turn)
            assert calls == (want if turn < 2 else []), (lens, turn)
            calls.clear()
            same = _step(plain, lens, 10 * i + turn)
            assert calls == want, lens
            # bfloat16 products by other kernels than those of a padded step
            assert ((got - same).norm() / same.norm()).item() < 2e-2, (lens, turn)
    again = _step(graphs, steps[1][0], 10)
    assert torch.equal(again, _step(graphs, steps[1][0], 10))  # the same graph between others of its shape
