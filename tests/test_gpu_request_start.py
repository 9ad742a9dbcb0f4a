"""A request's first state on the device: a slot's rows zeroed, the sampler's state set, each in one launch."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def test_a_slot_s_rows_of_every_tensor_and_no_others_are_zeroed():
    from oracle_engine_b200.cache.state import StateStore
    from oracle_engine_b200.parts.spec import StateNeed
    store = StateStore(5, DEV)
    needs = {"big": ((3, 257, 129), torch.float32), "one": ((), torch.int32), "two": ((7,), torch.int64), "odd": ((3,), torch.float32),
             "half": ((6,), torch.bfloat16)}
    tensors = {n: store.add("part", n, StateNeed(s, d)) for n, (s, d) in needs.items()}
    for late in (False, True):
        if late:                                             # a tensor that comes later, of a row that is no multiple of 4 bytes
            tensors["late"] = store.add("part", "late", StateNeed((3,), torch.bfloat16))
        for slot in (0, 4, 2):
            for t in tensors.values():
                t.fill_(3)
            store.reset(slot)
            for t in tensors.values():
                assert (t[slot] == 0).all() and (t[[s for s in range(5) if s != slot]] == 3).all()
    with pytest.raises(IndexError):
        store.reset(5)


@pytest.mark.parametrize("n,penalty", [(1, 1.3), (2, 1.3), (100, 1.3), (257, 1.3), (600, 1.3), (100, 1.0)])
def test_the_sampler_s_state_at_a_sequence_s_start(n, penalty):
    from oracle_engine_b200.cache.state import StateStore
    from oracle_engine_b200.sampling.params import GenParams
    from oracle_engine_b200.sampling.sampler import HISTORY_CAPACITY, Sampler
    sampler = Sampler(StateStore(4, DEV), DEV)
    for t in (sampler.rng_seed, sampler.rng_counter, sampler.hist, sampler.hist_count):
        t.fill_(9)
    prompt = [1000 + i for i in range(n)]
    sampler.start_sequence(2, -(1 << 62) - 5, prompt, GenParams(repeat_penalty=penalty))
    assert sampler.rng_seed.tolist() == [9, 9, -(1 << 62) - 5, 9] and sampler.rng_counter.tolist() == [9, 9, 0, 9]
    recorded = prompt[:-1] if penalty > 1 else []
    assert sampler.hist_count.tolist() == [9, 9, len(recorded), 9]
    assert (sampler.hist[[0, 1, 3]] == 9).all()
    if recorded:
        want = [0] * HISTORY_CAPACITY
        for i, t in enumerate(recorded):
            want[i % HISTORY_CAPACITY] = t
        assert sampler.hist[2].tolist() == want
    with pytest.raises(OverflowError):
        sampler.start_sequence(0, 1 << 63, prompt, GenParams())
