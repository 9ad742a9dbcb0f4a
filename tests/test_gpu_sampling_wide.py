"""The sampler on wide rows (a cluster of blocks per row): the tokens of the plain chain in 64 bits."""
import pytest
import torch

import plain_llama as pl

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _edges(logits, temperature, top_k, top_p, u):
    """The tokens between which a draw within 1e-5 of u falls: sums of 32 bits may end on either side of an edge."""
    return {pl.sample(logits, temperature, top_k, top_p, min(max(u + d, 0.0), 1.0)) for d in (-1e-5, 0.0, 1e-5)}


@pytest.mark.parametrize("V", [8192, 8193, 32000, 32768, 32769, 100003, 131072])
@pytest.mark.parametrize("temperature,top_k,top_p,penalty", [(0.7, 40, 0.9, 1.15), (1.0, 0, 0.9, 1.0), (1.3, 0, 1.0, 1.3), (0.7, 1, 1.0, 1.0),
                                                             (1.0, 5000, 0.999, 1.0), (0.2, 0, 0.05, 1.0)])
def test_draws_are_those_of_the_plain_chain(V, temperature, top_k, top_p, penalty):
    from oracle_engine_b200.csrc import ops
    rows, cap = 3, 256
    g = torch.Generator().manual_seed(V + top_k)
    logits = torch.randn(rows, V, generator=g) * 3
    logits[:, 5:V:997] += 4                                    # a few that stand out
    seeds = torch.tensor([11, 1 << 40, 7, 3], dtype=torch.int64)
    counter = torch.tensor([0, 5, 1, 9], dtype=torch.int32)
    hist = torch.randint(0, V, (4, cap), generator=g).int()
    hist[:, 10:60] = hist[:, 0:1]                              # the same token many times
    hist_count = torch.tensor([30, 300, 0, 64], dtype=torch.int32)
    slots = [1, 0, 3]
    want = []
    for r, s in enumerate(slots):
        n = int(hist_count[s])
        ring = [int(hist[s, j % cap]) for j in range(max(0, n - cap), n)]
        x = pl.repeat_penalty(logits[r].double(), ring, penalty, 64)
        want.append(_edges(x, temperature, top_k, top_p, pl.uniform_from_counter(int(seeds[s]), int(counter[s]))))
    dev = [t.to(DEV) for t in (logits, seeds, counter, hist, hist_count)]
    out = torch.full((rows + 1,), -7, dtype=torch.int32, device=DEV)
    x = torch.cat([dev[0], dev[0][:1]])
    use = penalty > 1.0
    ops.sample_rows(x, out, torch.tensor(slots + [-1], dtype=torch.int32, device=DEV), temperature, top_k, top_p, penalty, 64, dev[1], dev[2],
                    dev[3] if use else None, dev[4] if use else None)
    got = out.tolist()
    assert got[rows] == -1                                     # a row without a slot
    for r in range(rows):
        assert got[r] in want[r], (r, got[r], want[r])
    assert dev[2].tolist() == [1, 6, 1, 10]                    # the draws are counted
    if use:
        for r, s in enumerate(slots):
            assert int(dev[4][s]) == int(hist_count[s]) + 1 and int(dev[3][s, int(hist_count[s]) % cap]) == got[r]


def test_rows_without_a_usable_logit_and_ties():
    from oracle_engine_b200.csrc import ops
    V = 40000
    x = torch.zeros(4, V)
    x[0] = float("nan")
    x[1, 777] = float("inf")
    x[2] = -float("inf")
    x[2, [100, 39999]] = 2.0                                   # a tie at the cut: both are kept
    x[3] = 1.0                                                 # all equal: top-k keeps all
    seeds, counter = torch.zeros(4, dtype=torch.int64, device=DEV), torch.zeros(4, dtype=torch.int32, device=DEV)
    slot = torch.arange(4, dtype=torch.int32, device=DEV)
    out = torch.empty(4, dtype=torch.int32, device=DEV)
    seen = set()
    for _ in range(20):
        ops.sample_rows(x.to(DEV), out, slot, 1.0, 1, 1.0, 1.0, 64, seeds, counter, None, None)
        got = out.tolist()
        assert got[0] == -1 and got[1] == -1                   # infinity minus infinity: no probability is a number
        assert got[2] in (100, 39999)
        u = pl.uniform_from_counter(0, int(counter[3]) - 1)
        assert abs(got[3] - int(u * V)) <= 1
        seen.add(got[2])
    assert seen == {100, 39999}
