"""The sampler's short way (a small top-k: few values at or above the k-th largest of the warps' maxima), and the rows that leave it."""
import pytest
import torch

import plain_llama as pl
from test_gpu_sampling_wide import DEV, _edges

pytestmark = pytest.mark.gpu


def _rows(V, g):
    """Logits whose large values lie anywhere, side by side, 512 apart (one thread's) and 32 together in one warp's places; few
    finite ones; one value that is no number."""
    x = torch.randn(6, V, generator=g) * 3
    x[1, V // 2:V // 2 + 300] += 9
    x[2, 7::512] += 9
    for j in range(0, V - 32, 512):
        x[3, j:j + 32] += 9
    x[4] = -float("inf")
    x[4, torch.randperm(V, generator=g)[:30]] = torch.randn(30, generator=g)
    x[5, 77] = float("nan")
    return x


@pytest.mark.parametrize("V", [8192, 32769, 128256])
@pytest.mark.parametrize("top_k,top_p", [(1, 1.0), (2, 0.5), (40, 0.9), (40, 1.0), (127, 0.999), (128, 0.9), (129, 0.9)])
def test_draws_of_a_small_top_k(V, top_k, top_p):
    from oracle_engine_b200.csrc import ops
    g = torch.Generator().manual_seed(V + top_k)
    x = _rows(V, g)
    rows = x.shape[0]
    seeds = torch.arange(rows, dtype=torch.int64) * 977 + top_k
    counter = torch.zeros(rows, dtype=torch.int32, device=DEV)
    slot = torch.arange(rows, dtype=torch.int32, device=DEV)
    out = torch.empty(rows, dtype=torch.int32, device=DEV)
    for draw in range(3):
        want = [_edges(x[r].double(), 0.8, top_k, top_p, pl.uniform_from_counter(int(seeds[r]), draw)) for r in range(rows - 1)]
        ops.sample_rows(x.to(DEV), out, slot, 0.8, top_k, top_p, 1.0, 64, seeds.to(DEV), counter, None, None)
        got = out.tolist()
        assert got[-1] == -1
        for r in range(rows - 1):
            assert got[r] in want[r], (draw, r, got[r], want[r])
