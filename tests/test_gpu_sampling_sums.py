"""Draws of the sampler's short way right beside the edge between two tokens: what the sums that decide them lose."""
import numpy as np
import pytest
import torch

import plain_llama as pl

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _close_draws(n, want):
    """Draw numbers of seed 0 whose uniform times n lies 2e-6 to 4e-6 beside a whole number."""
    c = np.arange(1, 1 << 24, dtype=np.uint64)
    z = (c + np.uint64(1)) * np.uint64(0x9E3779B97F4A7C15)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    m = (z ^ (z >> np.uint64(31))) >> np.uint64(40)
    rest = (m * np.uint64(n)) & np.uint64((1 << 24) - 1)
    near = ((rest > 34) & (rest < 67)) | ((rest > (1 << 24) - 67) & (rest < (1 << 24) - 34))
    return [int(v) for v in c[near][:want]]


@pytest.mark.parametrize("V,n", [(128256, 317), (128256, 53), (32000, 211)])
def test_equal_values_beside_an_edge(V, n):
    """n equal logits and nothing else: token floor(u n) of them.  Eight equal probabilities add up without rounding but for the run that
    ends at the token, whose at most seven err by 2^-24 each: 4e-7 of a token.  (Summed one after another in 32 bits all of them err by
    up to 1e-4 of one: an eighth to a half of these draws were other tokens.)"""
    from oracle_engine_b200.csrc import ops
    draws = _close_draws(n, 64)
    assert len(draws) == 64
    g = torch.Generator().manual_seed(n)
    x = torch.full((64, V), -float("inf"))
    places = torch.stack([torch.randperm(V, generator=g)[:n].sort().values for _ in draws])
    x.scatter_(1, places, 1.0)
    counter, slot = torch.tensor(draws, dtype=torch.int32, device=DEV), torch.arange(64, dtype=torch.int32, device=DEV)
    out = torch.empty(64, dtype=torch.int32, device=DEV)
    ops.sample_rows(x.to(DEV), out, slot, 1.0, 40, 1.0, 1.0, 64, torch.zeros(64, dtype=torch.int64, device=DEV), counter, None, None)
    want = [int(places[r, int(pl.uniform_from_counter(0, c) * n)]) for r, c in enumerate(draws)]
    assert out.tolist() == want
