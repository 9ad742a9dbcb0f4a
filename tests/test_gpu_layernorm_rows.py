"""The layer norm on both sides of the rows up to which gains and shifts are read before the wait."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("rows", [1, 148, 149, 256, 257])
@pytest.mark.parametrize("D", [4, 2044, 8192, 8196])
def test_both_sides_of_the_line(rows, D):
    from oracle_engine_b200.csrc import build, ops
    few = build.load("elementwise").oe_layernorm_bf16_few
    assert [n for n in (1, 148, 149, 256, 257) if few(n)] == [1, 148]      # a block of 512 threads and 124 registers an SM
    g = torch.Generator(device=DEV).manual_seed(rows + D)
    x, w, b = torch.randn(rows, D, generator=g, device=DEV), torch.randn(D, generator=g, device=DEV), torch.randn(D, generator=g, device=DEV)
    y = torch.full((rows + 1, D), 7.0, dtype=torch.bfloat16, device=DEV)
    ops.layernorm(y[:rows], x, w, b, 1e-5)
    v = x.double()
    want = (v - v.mean(1, keepdim=True)) / (v.var(1, unbiased=False, keepdim=True) + 1e-5).sqrt() * w.double() + b.double()
    # one bfloat16 rounding (2^-9) of float32 sums of D values
    assert ((y[:rows].double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all() and (y[rows] == 7.0).all()
