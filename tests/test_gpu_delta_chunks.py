"""The gated delta rule in chunks against the recurrence walked token by token, in 64 bits."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _recurrence(qkv, gb, S, G, H, dk, dv):
    q, k = qkv[:, :G * dk].view(-1, G, dk), qkv[:, G * dk:2 * G * dk].view(-1, G, dk)
    q, k = q.repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1)
    v = qkv[:, 2 * G * dk:].view(-1, H, dv)
    out = torch.zeros_like(v)
    for t in range(v.shape[0]):
        S = gb[t, :H, None, None] * S
        u = gb[t, H:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None, :]
        out[t] = torch.einsum("hkv,hk->hv", S, q[t])
    return out.reshape(-1, H * dv), S


@pytest.mark.parametrize("G,H,dk,dv", [(1, 1, 64, 16), (2, 4, 128, 128), (1, 3, 128, 48), (3, 3, 64, 80)])
@pytest.mark.parametrize("lens", [[1], [32], [33, 1, 31], [64, 200, 2, 95]])
@pytest.mark.parametrize("decay", ["gentle", "hard"])
def test_chunks_are_the_recurrence(G, H, dk, dv, lens, decay):
    from oracle_engine_b200.csrc import ops
    g = torch.Generator().manual_seed(H * 1000 + sum(lens))
    T, C, slots = sum(lens), 2 * G * dk + H * dv, 9
    qkv = torch.randn(T + 5, C, generator=g)
    qk = qkv[:, :2 * G * dk].view(-1, 2 * G, dk)
    qk /= qk.norm(dim=-1, keepdim=True)                     # unit vectors, as the mixer's are
    gb = torch.rand(T + 5, 2 * H, generator=g)
    gb[:, :H] = 1 - 0.1 * gb[:, :H] if decay == "gentle" else gb[:, :H] ** 30         # from near one to zero (underflow)
    state = torch.randn(slots, H, dk, dv, generator=g)
    slot = torch.randperm(slots, generator=g)[:len(lens)].tolist()
    # a padding sequence in front of the last one, without a slot and without tokens
    cu, order = [0], []
    for i, n in enumerate(lens):
        if i == len(lens) - 1:
            order.append(-1)
            cu.append(cu[-1])
        order.append(slot[i])
        cu.append(cu[-1] + n)
    ctx = SimpleNamespace(n_seqs=len(order), n_tokens=T + 5, seq_slot=torch.tensor(order, dtype=torch.int32, device=DEV),
                          cu_q=torch.tensor(cu, dtype=torch.int32, device=DEV))
    S, o = state.to(DEV), torch.full((T + 5, H * dv), 7.0, device=DEV)
    assert ops.delta_chunks_supported(G, H, dk, dv)
    blocks = torch.empty(ops.delta_chunks_floats(ctx, H, dk, dv), device=DEV)
    ops.delta_chunks(o, S, blocks, qkv.to(DEV), gb.to(DEV), ctx, G, H, dk, dv)
    Sw, ow = state.clone().to(DEV), torch.zeros(T + 5, H * dv, device=DEV)
    ops.delta_rule_scan(ow, Sw, qkv.to(DEV), gb.to(DEV), ctx, G, H, dk, dv)
    at = 0
    for i, n in enumerate(lens):
        out, end = _recurrence(qkv[at:at + n].double(), gb[at:at + n].double(), state[slot[i]].double(), G, H, dk, dv)
        rel = lambda a, b: ((a.double().cpu() - b).norm() / b.norm()).item()                 # noqa: E731
        mine, walked = rel(o[at:at + n], out), rel(ow[at:at + n], out)
        # float32 sums of dk products and of 32 tokens; no further off than a few times the walk token by token
        assert mine < 2e-6 and mine < 4 * walked + 2e-7, (mine, walked)
        assert rel(S[slot[i]], end) < 2e-6
        at += n
    rest = [s for s in range(slots) if s not in slot]
    assert torch.equal(S[rest].cpu(), state[rest])
    assert (o[T:] == 7.0).all()


def test_an_infinite_value_does_not_reach_the_tokens_before_it():
    from oracle_engine_b200.csrc import ops
    G, H, dk, dv, T = 1, 1, 64, 16, 40
    g = torch.Generator().manual_seed(5)
    qkv, gb = torch.randn(T, 2 * dk + dv, generator=g) * 0.1, torch.rand(T, 2, generator=g)
    qkv[21, 2 * dk:] = float("inf")
    ctx = SimpleNamespace(n_seqs=1, n_tokens=T, seq_slot=torch.zeros(1, dtype=torch.int32, device=DEV),
                          cu_q=torch.tensor([0, T], dtype=torch.int32, device=DEV))
    S, o = torch.zeros(1, H, dk, dv, device=DEV), torch.zeros(T, dv, device=DEV)
    ops.delta_chunks(o, S, torch.empty(ops.delta_chunks_floats(ctx, H, dk, dv), device=DEV), qkv.to(DEV), gb.to(DEV), ctx, G, H, dk, dv)
    assert torch.isfinite(o[:21]).all() and not torch.isfinite(o[21:]).any()
