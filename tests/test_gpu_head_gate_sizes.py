"""The gate of a head's outputs at the edges of what a lane keeps (2, 4, 8 values; heads of any size above 256)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dv", [1, 33, 64, 65, 128, 129, 256, 257, 512])
@pytest.mark.parametrize("T,H", [(1, 1), (3, 5), (300, 4)])
@pytest.mark.parametrize("norm,wide", [(True, False), (True, True), (False, None)])
def test_against_64_bits(dv, T, H, norm, wide):
    from oracle_engine_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(dv + T)
    o, gate = torch.randn(T, H * dv, generator=g, device=DEV), torch.randn(T, H * dv + 3, generator=g, device=DEV)
    w = None if wide is None else torch.randn(H * dv if wide else dv, generator=g, device=DEV)
    out = torch.full((T + 1, H * dv), 7.0, device=DEV)
    ops.head_gate(out[:T], o, gate[:, :H * dv], w, H, dv, norm, "silu", 1e-5)
    v, z = o.double().view(T, H, dv), gate[:, :H * dv].double().view(T, H, dv)
    if norm:
        v = v / (v.square().mean(-1, keepdim=True) + 1e-5).sqrt()
    if w is not None:
        v = v * (w.double().view(H, dv) if wide else w.double())
    want = (v * z * torch.sigmoid(z)).reshape(T, H * dv)
    # float32 throughout: a sum of dv squares, an exponential and a few products
    assert ((out[:T].double() - want).abs() <= 4e-6 * want.abs() + 1e-7).all() and (out[T] == 7.0).all()
    same = o.clone()
    ops.head_gate(same, same, gate[:, :H * dv], w, H, dv, norm, "silu", 1e-5)          # in place
    assert torch.equal(same, out[:T])
