"""The prompt attention's grid that lists the tiles there are, and the grid of sequences by tiles: the same bits."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("hd,H,KVH", [(128, 24, 8), (64, 8, 2)])
@pytest.mark.parametrize("cluster", [1, 2, 8])
def test_both_grids(hd, H, KVH, cluster, monkeypatch):
    """As many SMs as list all tiles, and one SM, with which nothing is listed; rows that belong to no sequence stay as they are."""
    from oracle_engine_b200.csrc import ops, ops_tc
    qlens, starts, T = [70, 0, 1, 131, 0, 33], [600, 0, 300, 62, 0, 0], 256
    B, pages = len(qlens), 12
    g = torch.Generator(device=DEV).manual_seed(hd + cluster)
    cache = torch.randn(B * pages, 2, KVH, 64, hd, generator=g, device=DEV).bfloat16()
    tables = torch.randperm(B * pages, generator=torch.Generator().manual_seed(2)).int().view(B, pages).to(DEV)
    qkv = torch.randn(T, (H + 2 * KVH) * hd, generator=g, device=DEV).bfloat16()
    cu = [0]
    for q in qlens:
        cu.append(cu[-1] + q)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)                  # noqa: E731
    ctx = SimpleNamespace(n_seqs=B, max_qlen=T, cu_q=i32(cu), seq_start=i32(starts), seq_qlen=i32(qlens), all_decode=False, tok_seq=None)
    got = []
    for sms in (4096, 1):
        monkeypatch.setattr(ops, "sm_count", lambda: sms)                          # noqa: B023
        out = torch.full((T, H * hd), 7.0, dtype=torch.bfloat16, device=DEV)
        with ops_tc.knobs(prompt_cluster=cluster):
            ops_tc.attention(out, qkv, cache, tables, ctx, H, KVH, hd, 0, hd ** -0.5)
        got.append(out)
    assert ops_tc.device_error() == 0
    assert torch.equal(got[0], got[1]) and (got[0][cu[-1]:] == 7.0).all() and (got[0][:cu[-1]] != 7.0).any()
