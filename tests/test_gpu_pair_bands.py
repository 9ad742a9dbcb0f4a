"""The two-SM product over more row tiles than a band holds: every tile is computed once, in any order."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("M", [8 * 256, 8 * 256 + 1, 9 * 256, 17 * 256 - 5])
@pytest.mark.parametrize("N", [96, 1000])
def test_bands_of_row_tiles(M, N):
    from oracle_engine_b200.csrc import ops_tc
    K = 136
    g = torch.Generator(device=DEV).manual_seed(M + N)
    a = torch.randn(M, K, generator=g, device=DEV).bfloat16()
    w = torch.randn(N, K, generator=g, device=DEV).bfloat16()
    base = torch.randn(M, N, generator=g, device=DEV)
    want = a.double() @ w.double().T
    bound = K * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T) + 1e-6
    out = torch.full((M, N), float("nan"), device=DEV)
    ops_tc.gemm(out, a, w, kernel="pair")
    assert ((out.double() - want).abs() <= bound).all()
    acc = base.clone()
    ops_tc.gemm(acc, a, w, accumulate=True, kernel="pair")       # added once
    assert ((acc.double() - base.double() - want).abs() <= bound + 2.0 ** -22 * (base.abs() + want.abs())).all()
    assert ops_tc.device_error() == 0


@pytest.mark.parametrize("M", [8 * 256, 8 * 256 + 1, 9 * 256, 17 * 256 - 5])
@pytest.mark.parametrize("N,K", [(96, 136), (1000, 136), (400, 272), (700, 1024)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_either_order_of_the_tiles_gives_the_bits_of_the_one_sm_kernel_with_whole_tiles(M, N, K, dtype):
    """Wide weights with all rows first (1,000 rows of 136), the others in bands, of one and of several columns of tiles."""
    from oracle_engine_b200.csrc import ops_tc
    g = torch.Generator(device=DEV).manual_seed(M + N)
    a = torch.randn(M, K, generator=g, device=DEV).bfloat16()
    w = torch.randn(N, K, generator=g, device=DEV).bfloat16()
    one, two = (torch.empty(M, N, dtype=dtype, device=DEV) for _ in range(2))
    ops_tc.gemm(one, a, w, kernel="tcgen05", split_k=False)
    ops_tc.gemm(two, a, w, kernel="pair")
    assert torch.equal(one, two) and ops_tc.device_error() == 0


@pytest.mark.parametrize("M", [3314, 3315])
def test_activations_on_either_side_of_what_the_l2_keeps(M):
    """13 row tiles of 8,448 k and wide weights: up to 56 MB all rows first, beyond in bands."""
    from oracle_engine_b200.csrc import ops_tc
    N, K = 12800, 8448
    g = torch.Generator(device=DEV).manual_seed(M)
    a = torch.randn(M, K, generator=g, device=DEV).bfloat16()
    w = torch.randn(N, K, generator=g, device=DEV).bfloat16()
    one, two = (torch.empty(M, N, device=DEV) for _ in range(2))
    ops_tc.gemm(one, a, w, kernel="tcgen05", split_k=False)
    ops_tc.gemm(two, a, w, kernel="pair")
    assert torch.equal(one, two) and ops_tc.device_error() == 0
