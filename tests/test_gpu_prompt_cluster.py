"""The tcgen05 prompt attention whose tiles' pages are shared by the CTAs of a cluster, and the grid that lists the tiles there are."""
import math
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("hd,H,KVH", [(128, 24, 8), (64, 8, 2), (128, 5, 1)])
@pytest.mark.parametrize("window,sink", [(0, False), (100, True), (-150, False)])
@pytest.mark.parametrize("cluster", [1, 2, 4, 8])
def test_shared_pages(hd, H, KVH, window, sink, cluster):
    """Sequences of 1 page to 20, tiles with fewer pages than ranks, padding sequences between and behind them, windows that leave
    ranks without a key; against 64 bits, with the bounds of the unshared kernel: P and the output are bfloat16 (2^-9 each)."""
    from oracle_engine_b200.csrc import ops, ops_tc
    qlens, starts = [70, 0, 1, 131, 33], [1200, 0, 300, 62, 0]
    G, B, T = H // KVH, len(qlens), sum(qlens)
    g = torch.Generator(device=DEV).manual_seed(hd + H + cluster)
    pages = [(q + s + 63) // 64 for q, s in zip(qlens, starts)]
    tables = torch.full((B, 24), -1, dtype=torch.int32)
    order = torch.randperm(sum(pages), generator=torch.Generator().manual_seed(1)).tolist()
    for b, n in enumerate(pages):
        tables[b, :n] = torch.tensor([order.pop() for _ in range(n)], dtype=torch.int32)
    cache = torch.randn(sum(pages), 2, KVH, 64, hd, generator=g, device=DEV).bfloat16()
    qkv = torch.randn(T, (H + 2 * KVH) * hd, generator=g, device=DEV).bfloat16()
    cu = [0]
    for q in qlens:
        cu.append(cu[-1] + q)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)                  # noqa: E731
    ctx = SimpleNamespace(n_seqs=B, max_qlen=T, cu_q=i32(cu), seq_start=i32(starts), seq_qlen=i32(qlens), all_decode=False, tok_seq=None)
    out = torch.full((T, H * hd), 7.0, dtype=torch.bfloat16, device=DEV)
    with ops_tc.knobs(prompt_cluster=cluster):
        ops_tc.attention(out, qkv, cache, tables.to(DEV), ctx, H, KVH, hd, window, hd ** -0.5, sink)
    assert ops_tc.device_error() == 0
    for b in range(B):
        if not qlens[b]:
            continue
        kv = cache[tables[b, :pages[b]].long().to(DEV)].double().permute(1, 2, 0, 3, 4).reshape(2, KVH, -1, hd)
        n = starts[b] + qlens[b]
        q = qkv[cu[b]:cu[b + 1], :H * hd].double().view(-1, KVH, G, hd)
        s = torch.einsum("tkgd,knd->tkgn", q, kv[0, :, :n]) * hd ** -0.5
        pos = torch.arange(starts[b], n, device=DEV)[:, None]
        key = torch.arange(n, device=DEV)[None]
        seen = key <= pos
        if window > 0:
            seen &= pos - key < window
        elif window < 0:
            seen &= key // -window == pos // -window
        s = s.masked_fill(~seen[:, None, None], -math.inf)
        top = s.amax(-1, keepdim=True).clamp(min=0.0 if sink else -math.inf)
        p = torch.exp(s - top)
        weight = p / (p.sum(-1, keepdim=True) + (torch.exp(-top) if sink else 0.0))
        want = torch.einsum("tkgn,knd->tkgd", weight, kv[1, :, :n]).reshape(-1, H * hd)
        bound = 2.0 ** -8 * torch.einsum("tkgn,knd->tkgd", weight, kv[1, :, :n].abs()).reshape(-1, H * hd) + 2.0 ** -8 * want.abs() + 1e-4
        assert ((out[cu[b]:cu[b + 1]].double() - want).abs() <= bound).all()


def test_the_rule():
    from oracle_engine_b200.csrc import ops_tc
    rule = lambda t, b, cls, group=3, kvh=8: ops_tc.prompt_cluster(t, b, group, kvh, cls, sm_count=148)      # noqa: E731
    assert [rule(t, 1, 0) for t in (64, 256, 2048)] == [1, 1, 1]
    assert [rule(t, 1, 1) for t in (64, 128, 256, 500, 800, 2048)] == [8, 4, 2, 2, 1, 1] and rule(256, 8, 2) == 2 and rule(256, 16, 3) == 1
