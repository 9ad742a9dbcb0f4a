"""What a request's start does on the host: ids as an array, pages taken and given back many at a time."""
import random

import numpy as np
import pytest

from oracle_engine_b200.cache.slots import CacheFull, PagePool
from oracle_engine_b200.engine.step import _id_array


def test_many_pages_at_once_are_those_of_one_call_each():
    rng = random.Random(3)
    one, many = PagePool(40), PagePool(40)
    held: list = []
    for _ in range(300):
        if held and rng.random() < 0.5:
            rng.shuffle(held)
            n = rng.randint(1, len(held))
            back, held = held[:n], held[n:]
            for p in back:
                one.release(p)
            many.release_all(back)
        else:
            n = rng.randint(0, one.n_free)
            pages = [one.alloc() for _ in range(n)]
            assert many.alloc_many(n) == pages
            held += pages
        assert one._free == many._free and one._used == many._used
        many.check()


def test_many_pages_at_once_refuse_what_one_call_refuses():
    pool = PagePool(3)
    with pytest.raises(CacheFull):
        pool.alloc_many(4)
    assert pool.alloc_many(2) == [0, 1] and pool.n_free == 1
    for wrong in ([0, 2], [0, 0]):
        with pytest.raises(ValueError):
            pool.release_all(wrong)
    assert pool.n_free == 1                                  # nothing was given back
    pool.release_all([1, 0])
    pool.check()


def test_ids_of_any_kind_become_the_array_that_numpy_makes():
    for tokens in ([1, 2, 3], [np.int64(5), 7, True], [2 ** 31 - 1, -2 ** 31], [1.9, 2.0], np.arange(5), (4, 5), [2 ** 40, 1], [[1, 2], [3, 4]]):
        got, want = _id_array(tokens), np.asarray(tokens, dtype=np.int64)
        assert got.shape == want.shape and (got == want).all()
    for tokens in (["a"], [None]):
        with pytest.raises((TypeError, ValueError)):
            _id_array(tokens)


@pytest.mark.parametrize("n", [1, 2, 100, 257, 600])
def test_a_sequence_s_start_records_prompts_of_any_kind(n):
    """On the host as on the device; the ids may come in whatever int() takes them from."""
    import torch

    from oracle_engine_b200.cache.state import StateStore
    from oracle_engine_b200.sampling.params import GenParams
    from oracle_engine_b200.sampling.sampler import HISTORY_CAPACITY, Sampler
    ids = [7 * i % 1000 for i in range(n)]
    want = [0] * HISTORY_CAPACITY
    for i, t in enumerate(ids[:-1]):
        want[i % HISTORY_CAPACITY] = t
    for prompt in (ids, tuple(ids), np.asarray(ids), np.asarray(ids, dtype=np.int16), torch.tensor(ids), [torch.tensor(i) for i in ids],
                   [float(i) for i in ids], [str(i) for i in ids]):
        sampler = Sampler(StateStore(3, "cpu"), "cpu")
        sampler.hist.fill_(5)
        sampler.start_sequence(1, -9, prompt, GenParams())
        assert (int(sampler.rng_seed[1]), int(sampler.rng_counter[1]), int(sampler.hist_count[1])) == (-9, 0, n - 1)
        assert sampler.hist[1].tolist() == (want if n > 1 else [5] * HISTORY_CAPACITY) and (sampler.hist[[0, 2]] == 5).all()


def test_ids_that_do_not_fit_are_not_recorded_as_others():
    from oracle_engine_b200.cache.state import StateStore
    from oracle_engine_b200.sampling.params import GenParams
    from oracle_engine_b200.sampling.sampler import Sampler
    for prompt in ([2 ** 32 + 5, 1], np.asarray([2 ** 32 + 5, 1])):
        with pytest.raises(OverflowError):
            Sampler(StateStore(1, "cpu"), "cpu").start_sequence(0, 1, prompt, GenParams())
