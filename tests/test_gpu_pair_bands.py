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
    one = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    ops_tc.gemm(one, a, w, kernel="tcgen05")
    two = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    ops_tc.gemm(two, a, w, kernel="pair")
    assert torch.equal(one, two) or ((one.double() - two.double()).abs() <= 2.0 ** -7 * want.abs() + 1e-6).all()
    assert ops_tc.device_error() == 0
