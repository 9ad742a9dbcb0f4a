"""Which steps start their kernels early."""
import pytest

import fovirax_models
import fuvipel_models
import goridra_models

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("design,mixture", [("fovirax", True), ("goridra", True), ("fuvipel", False)])
def test_long_steps_of_a_mixture_start_nothing_early(design, mixture, tmp_path, monkeypatch):
    from oracle_engine_b200.csrc import build
    from oracle_engine_b200.engine.batch import SequenceStep
    from oracle_engine_b200.engine.engine import Engine
    models = {"fovirax": fovirax_models, "goridra": goridra_models, "fuvipel": fuvipel_models}[design]
    eng = Engine.from_pretrained(models.write(tmp_path, models.REAL, 11), dtype="bfloat16", max_tokens=2048)
    assert eng.model.has_mixture == mixture
    seen, switch = [], build.set_early_launch
    monkeypatch.setattr(build, "set_early_launch", lambda on: (seen.append(on), switch(on)))
    for tokens, calm in ((256, False), (257, mixture), (512, mixture), (513, True)):
        slot = eng.alloc()
        seen.clear()
        eng.step([SequenceStep(slot, [t % 90 for t in range(tokens)], [tokens - 1])])
        assert seen == ([False, True] if calm else []), tokens
        assert build._early_launch == [True]
        eng.free(slot)
