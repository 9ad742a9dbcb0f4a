"""Which scan a step's recurrent layers take, by the lengths of its sequences."""
import pytest
import torch

import fuvipel_models
from oracle_engine_b200.engine.batch import SequenceStep, StepBuffers, build_plan
from oracle_engine_b200.parts import delta_rule, time_mix


def _plan(lens, **kw):
    return build_plan([SequenceStep(i, [1] * n) for i, n in enumerate(lens)], [0] * len(lens), **kw)


def test_a_plan_says_its_real_lengths_whatever_the_padding():
    for lens in ([5], [1, 1, 1], [32, 33, 64, 200, 1]):
        for pad in ({}, {"pad_seqs": 16, "pad_tokens": 512}):
            plan = _plan(lens, **pad)
            plan.max_qlen = plan.n_tokens                     # as a captured step does
            ctx = StepBuffers(plan.n_tokens, plan.n_seqs, 0, [], "cpu").upload(plan, [])
            for step in (plan, ctx):
                assert (step.longest, step.scan_chunks) == (max(lens), sum(-(-n // 32) for n in lens))
                assert step.n_real_tokens == sum(lens)


def _delta(lens, heads, dv=128, padded=None):
    p = _plan(lens)
    return delta_rule.chunked(padded or p.n_tokens, p.longest, p.scan_chunks, heads, dv)


def _decay(lens, heads, d):
    p = _plan(lens)
    return time_mix.chunked(p.n_tokens, p.n_real_tokens, p.longest, p.scan_chunks, heads, d)


@pytest.mark.parametrize("heads,dv,walk,chunks", [
    (16, 128, [[32], [64], [5] * 8, [40] * 32, [300] * 4, [300] * 8, [192] + [1] * 31, [1] * 63 + [1000]],
     [[96], [256], [1111], [4096], [4096, 1, 1, 1]]),
    (8, 128, [[64], [5] * 8, [300] * 8, [1000] * 8, [192] + [1] * 31, [1] * 63 + [1000]],
     [[128], [300] * 2, [1000] * 2, [192] + [1] * 7, [1000] + [1] * 31, [1000, 500, 250, 125]]),
    (24, 128, [[64], [256], [1000] * 2, [300] * 8], []),
    (16, 64, [[64], [300] * 8, [40] * 32, [192] + [1] * 31], [[128], [1111], [1000] + [1] * 31])])
def test_the_delta_rule_goes_in_chunks_where_they_measured_faster(heads, dv, walk, chunks):
    assert not any(_delta(l, heads, dv) for l in walk) and all(_delta(l, heads, dv) for l in chunks)
    assert not _delta([300], heads, dv, padded=delta_rule.CHUNKS_MAX_TOKENS + 1)


@pytest.mark.parametrize("heads,d,walk,chunks", [
    (32, 64, [[32], [64], [5] * 8, [300] * 8, [64] * 16, [40] * 32, [192] + [1] * 31],
     [[96], [1111], [300] * 2, [192] + [1] * 7, [1000] + [1] * 31, [4096, 1, 1, 1]]),
    (16, 64, [[64], [300] * 16, [40] * 32], [[96], [300] * 4, [1000] + [1] * 31]),
    (8, 128, [[48], [5] * 8, [20] * 8], [[64], [1111], [300] * 8, [64] * 16, [300] * 32, [192] + [1] * 31]),
    (16, 128, [[48], [20] * 8, [192] + [1] * 31], [[64], [300] * 16, [1000] + [1] * 31])])
def test_the_time_mixing_goes_in_chunks_where_they_measured_faster(heads, d, walk, chunks):
    assert not any(_decay(l, heads, d) for l in walk) and all(_decay(l, heads, d) for l in chunks)


def test_steps_of_one_padded_shape_and_other_scans_have_other_keys():
    from oracle_engine_b200.config.fuvipel import FuvipelConfig
    from oracle_engine_b200.config.base import get_architecture
    from oracle_engine_b200.engine.runtime import Runtime
    from oracle_engine_b200.parts.model import DecoderModel
    arch = get_architecture("Fuvipel")
    model = DecoderModel(arch.build_spec(FuvipelConfig.from_dict(fuvipel_models.REAL)), Runtime(torch.bfloat16, torch.device("cpu")))
    for mixer in [model.layers[1].mixer] + [m for i in (0, 2) for _, m, _ in model.layers[i].mixer.branches]:
        if hasattr(mixer, "chunks"):
            mixer.chunks = True                               # as on the device
    steps = {"long": [200] + [1] * 3, "short": [50] * 4, "one": [250], "few": [60] * 4}
    choice = {n: model.step_choice(_plan(lens, pad_seqs=4, pad_tokens=256)) for n, lens in steps.items()}
    assert choice["short"] == choice["few"] != choice["long"] == choice["one"]
    assert choice["long"] == ((None, True), True, (None, True)) and choice["short"] == ((None, False), False, (None, False))


def test_a_branch_that_says_nothing_of_its_choice_chooses_nothing():
    """A mixer needs what the interface names; it need not derive from Part."""
    from types import SimpleNamespace

    from oracle_engine_b200.engine.runtime import Runtime
    from oracle_engine_b200.parts import parallel
    from oracle_engine_b200.parts.registry import MIXERS

    @MIXERS.register("says_nothing")
    class SaysNothing:
        def __init__(self, params, prefix, runtime):
            pass

        def cache_need(self):
            return None
    branches = [{"tag": t, "kind": "says_nothing", "prefix": t, "params": {}, "coef": 1.0} for t in "ab"]
    try:
        both = parallel.ParallelMixers({"hidden_size": 8, "branches": branches}, "", Runtime(torch.bfloat16, torch.device("cpu")))
        assert both.step_choice(SimpleNamespace(n_tokens=3, longest=3, scan_chunks=1, n_real_tokens=3)) == (None, None)
    finally:
        MIXERS.unregister("says_nothing")
