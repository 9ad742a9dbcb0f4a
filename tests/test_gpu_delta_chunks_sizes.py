"""The delta rule in chunks on both sides of a block an SM, for the chunks' systems and for the scan: the same bits."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("H,dk,dv", [(4, 64, 64), (4, 128, 16)])
def test_a_sequence_among_others_is_the_sequence_alone(H, dk, dv):
    """One sequence is 12 blocks of systems and 16 (or 4) of the scan; 16 and 40 of them are more than the device has SMs for, at
    two and at three blocks an SM."""
    from oracle_engine_b200.csrc import ops
    n, most = 100, 40
    C = 2 * H * dk + H * dv
    g = torch.Generator(device=DEV).manual_seed(dk)
    qkv, gb = torch.randn(most * n, C, generator=g, device=DEV) * 0.1, torch.rand(most * n, 2 * H, generator=g, device=DEV)
    state = torch.randn(most, H, dk, dv, generator=g, device=DEV)

    def run(seqs):
        ctx = SimpleNamespace(n_seqs=len(seqs), n_tokens=n * len(seqs), seq_slot=torch.tensor(seqs, dtype=torch.int32, device=DEV),
                              cu_q=torch.arange(0, n * len(seqs) + 1, n, dtype=torch.int32, device=DEV))
        rows = torch.cat([torch.arange(s * n, s * n + n, device=DEV) for s in seqs])
        S, o = state.clone(), torch.empty(n * len(seqs), H * dv, device=DEV)
        blocks = torch.empty(ops.delta_chunks_floats(ctx, H, dk, dv), device=DEV)
        for _ in range(2):                                 # the second right behind the first
            S.copy_(state)
            ops.delta_chunks(o, S, blocks, qkv[rows], gb[rows], ctx, H, H, dk, dv)
        return o.view(len(seqs), n, -1), S

    alone = {s: run([s]) for s in (0, 7, 39)}
    for count in (12, 16, 40):
        o, S = run(list(range(count)))
        for s in (s for s in alone if s < count):
            assert torch.equal(o[s], alone[s][0][0]) and torch.equal(S[s], alone[s][1][s])
