"""The 32-bit products of a few rows (tiles of 16 weight rows, stages of 512 k): the bits of the general kernel."""
import pytest
import torch

from test_gpu_float32_path import DEV, _rand

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 2, 4, 5, 9, 48])
@pytest.mark.parametrize("N,K", [(1, 4), (16, 512), (17, 516), (2368, 1024), (2369, 1028), (31, 5120), (5000, 700)])
def test_a_few_rows_give_the_same_bits(M, N, K):
    """Edges of a tile (16), of a stage (512), of the ring (2, 4 and 5 stages, across tiles), of one CTA an SM (148 tiles: 2,368 rows);
    rows of A inside wider ones; accumulation; values that are no numbers stay in their row and column."""
    from oracle_engine_b200.csrc import ops
    a, w, base = _rand(M, K + 4, seed=1)[:, :K], _rand(N, K, seed=2), _rand(M, N, seed=3)
    a[M // 2, K - 1] = float("inf")
    w[N // 2, 0] = float("nan")
    plain, out = torch.empty(M, N, device=DEV), torch.full((M + 1, N), 7.0, device=DEV)
    ops.gemm_simple(plain, a, w, kind=4)
    ops.gemm_simple(out[:M], a, w, kind=1)
    assert torch.equal(out[:M].nan_to_num(nan=9.0), plain.nan_to_num(nan=9.0)) and (out[M] == 7.0).all()
    acc = base.clone()
    ops.gemm_simple(acc, a, w, accumulate=True, kind=1)
    assert torch.equal(acc.nan_to_num(nan=9.0), (base + plain).nan_to_num(nan=9.0))
