"""The gated delta rule's decode step in one launch against the kernels that a step of any tokens goes through."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("G,H,dk,dv,taps", [(8, 16, 128, 128, 4), (2, 2, 64, 64, 1), (1, 8, 32, 256, 2), (3, 9, 100, 36, 8), (2, 4, 6, 4, 3),
                                            (1, 1, 256, 64, 4)])
def test_the_step_in_one_launch(G, H, dk, dv, taps):
    from oracle_engine_b200.csrc import ops
    g = torch.Generator().manual_seed(G * 100 + dk)
    r = lambda *s: torch.randn(*s, generator=g).to(DEV)                                       # noqa: E731
    C, slots = 2 * G * dk + H * dv, 7
    P = C + H * dv + 2 * H
    slot = [3, -1, 0, 5]                                    # a padding sequence among them: no slot, no token
    proj = r(4, P)
    conv_w, A_log, dt_bias, norm_w = r(C, taps) * 0.5, r(H) * 0.3, r(H), 1 + 0.1 * r(dv)
    state, conv = r(slots, H, dk, dv), r(slots, max(taps - 1, 1), C)
    ctx = SimpleNamespace(n_seqs=4, n_tokens=4, seq_slot=torch.tensor(slot, dtype=torch.int32, device=DEV),
                          cu_q=torch.tensor([0, 1, 1, 2, 3], dtype=torch.int32, device=DEV),
                          tok_seq=torch.tensor([0, 2, 3, -1], dtype=torch.int32, device=DEV))
    S1, c1, S2, c2 = state.clone(), conv.clone(), state.clone(), conv.clone()
    qkv, gb = torch.zeros(4, C, device=DEV), torch.zeros(4, 2 * H, device=DEV)
    ops.short_conv_prepare(qkv, gb, proj, conv_w, c1, A_log, dt_bias, ctx, G, H, dk, dv, dk ** -0.5)
    ops.conv_state_update(c1, proj, C, taps, ctx)
    o = torch.zeros(4, H * dv, device=DEV)
    ops.delta_rule_scan(o, S1, qkv, gb, ctx, G, H, dk, dv)
    want = torch.zeros(4, H * dv, dtype=torch.bfloat16, device=DEV)
    ops.head_gate(want, o, proj[:, C:C + H * dv], norm_w, H, dv, True, "silu", 1e-6)
    y = torch.full((4, H * dv), 7.0, dtype=torch.bfloat16, device=DEV)
    assert ops.delta_step_supported(G, H, dk, dv, taps)
    ops.delta_step(y, S2, c2, proj, conv_w, A_log, dt_bias, norm_w, ctx, G, H, dk, dv, dk ** -0.5, 1e-6)
    assert torch.equal(c1, c2)                              # moved, not computed
    # float32 sums of dk products in another order, and the decay's own rounding
    assert ((S1 - S2).abs() <= 1e-5 * (1 + S1.abs())).all()
    used = [s for s in slot if s >= 0]
    rest = [s for s in range(slots) if s not in used]
    assert torch.equal(S2[rest], state[rest])
    # one bfloat16 rounding, of values that a norm may have scaled by how small the read-out is
    a, b = y[:3].float(), want[:3].float()
    assert ((a - b).abs() <= 2.0 ** -7 * b.abs() + 2e-3).all()
    assert (y[3] == 7.0).all()


@pytest.mark.parametrize("G,H,dk,dv,taps,seqs", [(8, 16, 128, 128, 4, 1), (8, 16, 128, 128, 4, 12), (1, 8, 32, 256, 2, 3)])
def test_steps_right_behind_one_another(G, H, dk, dv, taps, seqs):
    """A slot's reset and six tokens without anything between the launches: every step reads what the one before it wrote."""
    from oracle_engine_b200.csrc import ops
    g = torch.Generator().manual_seed(G + seqs)
    r = lambda *s: torch.randn(*s, generator=g).to(DEV)                                       # noqa: E731
    C, steps = 2 * G * dk + H * dv, 6
    P = C + H * dv + 2 * H
    proj, conv_w, A_log, dt_bias, norm_w = r(steps, seqs, P), r(C, taps) * 0.5, r(H) * 0.3, r(H), 1 + 0.1 * r(dv)
    state, conv = r(seqs, H, dk, dv), r(seqs, max(taps - 1, 1), C)
    ctx = SimpleNamespace(n_seqs=seqs, n_tokens=seqs, seq_slot=torch.arange(seqs, dtype=torch.int32, device=DEV),
                          cu_q=torch.arange(seqs + 1, dtype=torch.int32, device=DEV), tok_seq=torch.arange(seqs, dtype=torch.int32, device=DEV))
    S1, c1, S2, c2 = state.clone(), conv.clone(), state.clone(), conv.clone()
    want, y = torch.empty(2, steps, seqs, H * dv, dtype=torch.bfloat16, device=DEV)
    tables = [ops.row_table([S, c]) for S, c in ((S1, c1), (S2, c2))]
    qkv, gb, o = torch.zeros(seqs, C, device=DEV), torch.zeros(seqs, 2 * H, device=DEV), torch.zeros(seqs, H * dv, device=DEV)
    ops.zero_rows(*tables[0], 0)
    for i in range(steps):
        ops.short_conv_prepare(qkv, gb, proj[i], conv_w, c1, A_log, dt_bias, ctx, G, H, dk, dv, dk ** -0.5)
        ops.conv_state_update(c1, proj[i], C, taps, ctx)
        ops.delta_rule_scan(o, S1, qkv, gb, ctx, G, H, dk, dv)
        ops.head_gate(want[i], o, proj[i][:, C:C + H * dv], norm_w, H, dv, True, "silu", 1e-6)
    torch.cuda.synchronize()
    rows = [proj[i] for i in range(steps)]
    ops.zero_rows(*tables[1], 0)
    for i in range(steps):
        ops.delta_step(y[i], S2, c2, rows[i], conv_w, A_log, dt_bias, norm_w, ctx, G, H, dk, dv, dk ** -0.5, 1e-6)
    torch.cuda.synchronize()
    assert torch.equal(c1, c2)
    assert ((S1 - S2).abs() <= steps * 1e-5 * (1 + S1.abs())).all()       # as above, once a step
    a, b = y.float(), want.float()
    assert ((a - b).abs() <= 2.0 ** -7 * b.abs() + 4e-3).all()


def test_sizes_beyond_are_refused():
    from oracle_engine_b200.csrc import ops
    assert not ops.delta_step_supported(1, 9, 64, 64, 4)     # nine heads to a key head
    assert not ops.delta_step_supported(1, 1, 256, 128, 4)   # more rows than a thread keeps
    assert not ops.delta_step_supported(1, 1, 64, 66, 4) and not ops.delta_step_supported(1, 1, 64, 64, 9)
