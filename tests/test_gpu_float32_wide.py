"""Tiles of 128 x 128 of the 32-bit products: the bits of the general kernel."""
import pytest
import torch

from test_gpu_float32_path import DEV, _rand

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 65, 128, 129, 300])
@pytest.mark.parametrize("N,K", [(1, 516), (128, 512), (130, 516), (127, 1024), (300, 2052), (260, 1000), (257, 4)])
def test_tiles_of_128_give_the_same_bits(M, N, K):
    """Edges of tiles (128), of the one chain (512), of rounds of classes (512) and of stages (16); outputs whose rows are and are
    not 16-byte aligned; accumulation; values that are no numbers stay in their row and column."""
    from oracle_engine_b200.csrc import ops
    a, w, base = _rand(M, K, seed=1), _rand(N, K, seed=2), _rand(M, N + 3, seed=3)
    a[M // 2, K - 1] = float("inf")
    w[N // 2, 0] = float("nan")
    plain = torch.empty(M, N, device=DEV)
    ops.gemm_simple(plain, a, w, kind=4)
    for kind in (3,) if K <= 512 else (3, 5, 6):
        out = torch.full((M, N + 3), 7.0, device=DEV)
        ops.gemm_simple(out[:, :N], a, w, kind=kind)
        assert torch.equal(out[:, :N].nan_to_num(nan=9.0), plain.nan_to_num(nan=9.0)) and (out[:, N:] == 7.0).all()
        acc = base.clone()
        ops.gemm_simple(acc[:, :N], a, w, accumulate=True, kind=kind)
        assert torch.equal(acc[:, :N].nan_to_num(nan=9.0), (base[:, :N] + plain).nan_to_num(nan=9.0)) and torch.equal(acc[:, N:], base[:, N:])
    if K <= 512:
        with pytest.raises(ops.KernelError):
            ops.gemm_simple(plain, a, w, kind=5)
