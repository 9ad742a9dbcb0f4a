"""The decaying time mixing in chunks against the recurrence walked token by token, in 64 bits."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _recurrence(r, k, v, z, u, w0, S, H, d):
    r, k, v = (t.view(-1, H, d) for t in (r, k, v))
    w = torch.exp(-torch.exp(z + w0)).view(-1, H, d)
    out = torch.zeros_like(v)
    for t in range(v.shape[0]):
        kv = k[t][:, :, None] * v[t][:, None, :]
        out[t] = torch.einsum("hkv,hk->hv", S + u.view(H, d)[:, :, None] * kv, r[t])
        S = w[t][:, :, None] * S + kv
    return out.reshape(-1, H * d), S


@pytest.mark.parametrize("H,d", [(1, 64), (5, 64), (2, 128)])
@pytest.mark.parametrize("lens", [[1], [32], [33, 1, 31], [64, 200, 2, 95]])
@pytest.mark.parametrize("decay", [-4.0, 3.0])
def test_chunks_are_the_recurrence(H, d, lens, decay):
    from oracle_engine_b200.csrc import ops
    g = torch.Generator().manual_seed(H * 1000 + sum(lens))
    T, slots = sum(lens), 9
    rows = torch.randn(T + 5, 4 * H * d, generator=g)                       # r, k, v and z beside one another: a row stride
    u, w0 = torch.randn(H * d, generator=g), torch.randn(H * d, generator=g) + decay        # from hardly to within a few tokens
    state = torch.randn(slots, H, d, d, generator=g)
    slot = torch.randperm(slots, generator=g)[:len(lens)].tolist()
    cu, order = [0], []
    for i, n in enumerate(lens):
        if i == len(lens) - 1:                                              # a padding sequence: no slot, no token
            order.append(-1)
            cu.append(cu[-1])
        order.append(slot[i])
        cu.append(cu[-1] + n)
    ctx = SimpleNamespace(n_seqs=len(order), n_tokens=T + 5, seq_slot=torch.tensor(order, dtype=torch.int32, device=DEV),
                          cu_q=torch.tensor(cu, dtype=torch.int32, device=DEV))
    dev = rows.to(DEV)
    parts = [dev[:, i * H * d:(i + 1) * H * d] for i in range(4)]
    S, o = state.to(DEV), torch.full((T + 5, H * d), 7.0, device=DEV)
    ops.decay_chunks(o, S, torch.empty(ops.decay_chunks_floats(ctx, H, d), device=DEV), *parts, u.to(DEV), w0.to(DEV), ctx, H, d)
    Sw, ow = state.to(DEV), torch.zeros(T + 5, H * d, device=DEV)
    ops.decay_scan(ow, Sw, *parts, u.to(DEV), w0.to(DEV), ctx, H, d)
    at = 0
    for i, n in enumerate(lens):
        cut = [rows[at:at + n, j * H * d:(j + 1) * H * d].double() for j in range(4)]
        out, end = _recurrence(*cut, u.double(), w0.double(), state[slot[i]].double(), H, d)
        rel = lambda a, b: ((a.double().cpu() - b).norm() / b.norm()).item()                 # noqa: E731
        mine, walked = rel(o[at:at + n], out), rel(ow[at:at + n], out)
        assert mine < 2e-6 and mine < 4 * walked + 2e-7, (mine, walked)      # float32 sums in another order
        assert rel(S[slot[i]], end) < 2e-6
        at += n
    rest = [s for s in range(slots) if s not in slot]
    assert torch.equal(S[rest].cpu(), state[rest])
    assert (o[T:] == 7.0).all()


def test_an_infinite_value_does_not_reach_the_tokens_before_it():
    from oracle_engine_b200.csrc import ops
    d, T = 64, 40
    g = torch.Generator().manual_seed(5)
    r, k, v, z = (torch.randn(T, d, generator=g).to(DEV) for _ in range(4))
    v[21] = float("inf")
    ctx = SimpleNamespace(n_seqs=1, n_tokens=T, seq_slot=torch.zeros(1, dtype=torch.int32, device=DEV),
                          cu_q=torch.tensor([0, T], dtype=torch.int32, device=DEV))
    S, o, u = torch.zeros(1, 1, d, d, device=DEV), torch.zeros(T, d, device=DEV), torch.ones(d, device=DEV)
    ops.decay_chunks(o, S, torch.empty(ops.decay_chunks_floats(ctx, 1, d), device=DEV), r, k, v, z, u, u - 3, ctx, 1, d)
    assert torch.isfinite(o[:21]).all() and not torch.isfinite(o[21:]).any()
