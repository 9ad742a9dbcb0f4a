"""Which form a mixture's products take, by the numbers of tokens and experts: where each measured faster."""
import pytest

from oracle_engine_b200.parts import moe


@pytest.mark.parametrize("experts,top,stream,all_experts", [(8, 2, [1, 2, 4], [5, 6, 8, 16, 17]), (3, 1, [1, 3], [4]), (64, 8, [1, 8], [9, 16]),
                                                            (64, 2, [1, 16], [17]), (1, 1, [1], [2])])
def test_few_tokens_stream_the_chosen_experts(experts, top, stream, all_experts):
    assert all(moe._stream_pays(T, top, experts) for T in stream) and not any(moe._stream_pays(T, top, experts) for T in all_experts)


@pytest.mark.parametrize("D,ff,all_experts,by_expert", [(1024, 704, [330, 700, 1500, 2000], [6000]), (2048, 1408, [330, 512, 700, 1000], [1500, 2000, 16000]),
                                                        (3072, 2048, [330, 512, 700], [1000, 1500, 2000])])
def test_prompts_are_sorted_where_that_saves_enough(D, ff, all_experts, by_expert):
    assert not any(moe._sorted_pays(T, 2, 8, D, ff) for T in all_experts) and all(moe._sorted_pays(T, 2, 8, D, ff) for T in by_expert)


def test_a_mixture_of_which_every_token_takes_all_is_not_sorted():
    assert not moe._sorted_pays(100000, 4, 4, 8192, 8192) and not moe._sorted_pays(100000, 1, 1, 8192, 8192)
