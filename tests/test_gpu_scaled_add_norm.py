"""A scaled sublayer output added to the stream and the stream's norm, in one launch and apart."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("rows", [1, 5, 1300])
@pytest.mark.parametrize("D", [4, 100, 1024, 2052, 4096])
@pytest.mark.parametrize("two,scaled", [(False, False), (True, False), (False, True), (True, True)])
def test_one_launch_and_two(rows, D, two, scaled):
    from oracle_engine_b200.csrc import ops
    g = torch.Generator().manual_seed(rows + D)
    r = lambda *s: torch.randn(*s, generator=g).to(DEV)                                       # noqa: E731
    x, y0, y1, vec, w = r(rows, D), r(rows, D), r(rows, D), 1 + 0.1 * r(D), 1 + 0.1 * r(D)
    args = (vec if scaled else None, 0.75, 0.5, y1 if two else None, -1.25 if two else 0.0)
    want = x.double() + (vec.double() if scaled else 1.0) * 0.75 * (0.5 * y0.double() + (-1.25 * y1.double() if two else 0.0))
    apart = x.clone()
    ops.scaled_add(apart, y0, *args)
    assert ((apart.double() - want).abs() <= 4 * 2.0 ** -24 * (x.abs() + y0.abs() + 2 * y1.abs() + 1)).all()
    odd = torch.empty(rows, D + 1, device=DEV)[:, 1:].contiguous()           # another allocation of the same values
    odd.copy_(x)
    flat = torch.empty(rows * D + 1, device=DEV)[1:].view(rows, D)            # off a 16-byte boundary: a value a thread
    flat.copy_(x)
    ops.scaled_add(odd, y0, *args)
    ops.scaled_add(flat, y0, *args)
    assert torch.equal(odd, apart) and torch.equal(flat, apart)
    out, one = torch.empty(rows, D, dtype=torch.bfloat16, device=DEV), x.clone()
    ops.scaled_add_norm(out, one, y0, w, 1e-6, *args)
    assert torch.equal(one, apart)
    norm = want / torch.sqrt((want * want).mean(-1, keepdim=True) + 1e-6) * w.double()
    assert ((out.double() - norm).abs() <= 2.0 ** -8 * norm.abs() + 1e-5).all()
