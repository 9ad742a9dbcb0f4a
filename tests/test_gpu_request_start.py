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


def test_a_reset_goes_through_one_launch_where_rows_are_whole_words(monkeypatch):
    """Of few tensors as of many; a tensor added later is among the next reset's; rows of odd bytes are filled one by one."""
    from oracle_engine_b200.cache.state import StateStore
    from oracle_engine_b200.csrc import ops
    from oracle_engine_b200.parts.spec import StateNeed
    launches, zero_rows = [], ops.zero_rows
    monkeypatch.setattr(ops, "zero_rows", lambda *a: (launches.append(a[0].shape[0]), zero_rows(*a)))
    store, tensors, want = StateStore(3, DEV), [], []
    for i, (shape, dtype) in enumerate([((1,), torch.int32), ((4097,), torch.float32), ((2, 3), torch.bfloat16)] * 4 + [((5,), torch.bfloat16)]):
        tensors.append(store.add(i, "t", StateNeed(shape, dtype)))
        for t in tensors:
            t.fill_(3)
        store.reset(1)
        if i < 12:
            want.append(i + 1)
        assert launches == want
        for t in tensors:
            assert (t[1] == 0).all() and (t[[0, 2]] == 3).all()


@pytest.mark.parametrize("sizes", [[1], [4], [1023, 1, 70000], [2 ** 20 + 3] + [5] * 40])
def test_rows_of_a_table_are_zeroed(sizes):
    """Rows of one word and of more words than the pieces of the grid take at once, of many tensors; the rows around them stay."""
    from oracle_engine_b200.csrc import ops
    tensors = [torch.full((3, n), 7, dtype=torch.int32, device=DEV) for n in sizes]
    table, largest = ops.row_table(tensors)
    for row in (0, 2):
        ops.zero_rows(table, largest, row)
    for t in tensors:
        assert (t[[0, 2]] == 0).all() and (t[1] == 7).all()
    with pytest.raises(ops.KernelError):
        ops.row_table([torch.empty(2, 3, dtype=torch.bfloat16, device=DEV)])


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


def test_a_prompt_on_the_device_is_recorded_as_a_list_is():
    from oracle_engine_b200.cache.state import StateStore
    from oracle_engine_b200.sampling.params import GenParams
    from oracle_engine_b200.sampling.sampler import Sampler
    sampler = Sampler(StateStore(2, DEV), DEV)
    prompt = [3 * i for i in range(300)]
    sampler.start_sequence(0, 1, prompt, GenParams())
    sampler.start_sequence(1, 1, torch.tensor(prompt, device=DEV), GenParams())
    assert torch.equal(sampler.hist[0], sampler.hist[1]) and sampler.hist_count.tolist() == [299, 299]
