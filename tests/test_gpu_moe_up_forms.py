"""The two kernels of a mixture's up product: the same bits, and the rule between them."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("T", [1, 4, 8])
@pytest.mark.parametrize("D,E,ff,shared", [(256, 4, 32, 0), (2056, 8, 24, 16), (512, 8, 1024, 2048), (128, 64, 512, 512)])
def test_both_kernels_give_the_same_bits(T, D, E, ff, shared, monkeypatch):
    from oracle_engine_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(T + D)
    F, W = E * ff + shared, E + (1 if shared else 0)
    h, w = torch.randn(T, D, generator=g, device=DEV).bfloat16(), (torch.randn(2 * F, D, generator=g, device=DEV) * 0.05).bfloat16()
    dense = torch.zeros(T, W, device=DEV)
    for t in range(T - T // 4):                            # some tokens have no expert (padding)
        dense[t, [t % E, (3 * t + 1) % E]] = 0.5
        dense[t, E:] = 0.7
    got = []
    for ahead in (True, False):
        monkeypatch.setattr(ops, "moe_up_ahead", lambda *a, **k: ahead)                # noqa: B023
        a = torch.zeros(T, F, dtype=torch.bfloat16, device=DEV)
        for _ in range(2):
            ops.moe_up_stream(a, h, w, dense, E, ff)
        got.append(a)
    assert torch.equal(got[0], got[1]) and got[0].any()


def test_the_rule():
    from oracle_engine_b200.csrc import ops
    rule = lambda T, E, ff, shared, top=2: ops.moe_up_ahead(T, E * ff + shared, E, ff, top, sms=148)          # noqa: E731
    assert [rule(T, 8, 512, 512) for T in (1, 4, 8, 9)] == [True, True, True, False]
    assert [rule(T, 8, 1024, 2048) for T in (1, 2, 4)] == [True, False, False]
    assert [rule(T, 8, 1408, 0) for T in (1, 2, 4)] == [True, True, False] and not rule(1, 32, 1024, 0) and rule(1, 32, 128, 128) and not rule(1, 8, 1024, 0, top=8)
