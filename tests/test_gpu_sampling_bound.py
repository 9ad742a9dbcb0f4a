"""Draws of wide rows by the bound with many values at or above it: up to what is compared at once (512), and beyond."""
import pytest
import torch

import plain_llama as pl
from test_gpu_sampling_wide import DEV, _edges

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V,top_k", [(65536, 64), (128256, 117), (128256, 118), (8192, 32), (8193, 33)])
@pytest.mark.parametrize("top_p", [0.9, 1.0])
def test_draws_with_hundreds_of_values_at_the_bound(V, top_k, top_p):
    """Rows in any order (some 300 values at the last top-k that goes by the bound); one with as many equal values as fit, one with more."""
    from oracle_engine_b200.csrc import ops
    g = torch.Generator().manual_seed(V + top_k)
    x = torch.randn(4, V, generator=g) * 3
    places = torch.randperm(V, generator=g)
    equal = {1: 400, 2: 600, 3: V}                         # the largest values of a row: all are kept, whatever top-k and top-p say
    for r, n in equal.items():
        x[r, places[:n]] = 20.0
    seeds = torch.arange(4, dtype=torch.int64) * 31 + top_k
    counter, slot = torch.zeros(4, dtype=torch.int32, device=DEV), torch.arange(4, dtype=torch.int32, device=DEV)
    out = torch.empty(4, dtype=torch.int32, device=DEV)
    for draw in range(3):
        u = [pl.uniform_from_counter(int(s), draw) for s in seeds]
        ops.sample_rows(x.to(DEV), out, slot, 0.8, top_k, top_p, 1.0, 64, seeds.to(DEV), counter, None, None)
        got = out.tolist()
        assert got[0] in _edges(x[0].double(), 0.8, top_k, top_p, u[0]), draw
        for r, n in equal.items():
            kept = places[:n].sort().values.tolist()
            # sums of 32 bits over n equal values: less than one of them off among hundreds, 1e-5 of the mass among all
            assert abs(kept.index(got[r]) - int(u[r] * n)) <= 1 + 2e-5 * n, (draw, r, got[r])
