"""The kernels of the 32-bit path: products and attention whose results do not depend on the kernel that a shape goes to."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _rand(*shape, seed=0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(DEV)


@pytest.mark.parametrize("N,K", [(1, 4), (17, 60), (16, 64), (33, 68), (130, 512), (65, 516), (70, 508), (200, 1100), (4750, 576), (9500, 100)])
def test_products_give_the_same_bits_by_every_kernel(N, K):
    """Edges of the one chain (K = 512), of segments (64), of rounds of eight segments (512), of row tiles (16, 32, 64), of the tiles of rows of A
    (1, 2, 4, 8) and of the tiles of 64 and 128; rows of A inside wider ones; accumulation."""
    from oracle_engine_b200.csrc import ops
    w = _rand(N, K, seed=2)
    wide = _rand(140, K + 8, seed=1)
    base = _rand(140, N, seed=3)
    for M in (1, 2, 3, 5, 8, 9, 17, 33, 64, 65, 140):
        a = wide[:M, :K]
        want = a.double() @ w.double().T
        plain = torch.full((M, N), 7.0, device=DEV)
        ops.gemm_simple(plain, a, w, kind=4)
        # a chain of n additions has an error of at most n 2^-24 of the products' absolute sum; eight chains are added
        bound = (K + 1 if K <= 512 else K / 8 + 64 + 9) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)
        assert ((plain.double() - want).abs() <= bound).all()
        for kind in (0, 1, 2, 3):
            out = torch.full((M + 1, N), 7.0, device=DEV)
            ops.gemm_simple(out[:M], a, w, kind=kind)
            assert torch.equal(out[:M], plain), (M, N, K, kind)
            assert (out[M] == 7.0).all()
            acc = base[:M].clone()
            ops.gemm_simple(acc, a, w, accumulate=True, kind=kind)
            assert torch.equal(acc, base[:M] + plain), (M, N, K, kind)


def test_a_product_of_unaligned_rows_takes_the_general_kernel():
    from oracle_engine_b200.csrc import ops
    buf = _rand(5 * 64 + 1, seed=4)
    a, w = buf[1:].view(5, 64), _rand(40, 64, seed=5)
    out, same = torch.empty(5, 40, device=DEV), torch.empty(5, 40, device=DEV)
    ops.gemm_simple(out, a, w)
    ops.gemm_simple(same, a.clone(), w)
    assert torch.equal(out, same)
    with pytest.raises(ops.KernelError):
        ops.gemm_simple(out, a, w, kind=1)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,KVH,hd,window,sink", [(4, 2, 64, 0, False), (9, 1, 18, 0, True), (20, 2, 128, 40, False), (3, 3, 256, -50, True),
                                                  (2, 1, 34, 1, False), (33, 1, 16, 0, False)])
def test_attention_gives_the_same_bits_by_both_kernels(dtype, H, KVH, hd, window, sink):
    """Chunks of 32 keys at their edges, more heads a group than a warp takes at a time, windows and chunks of positions,
    padding rows; the values that a query does not see are infinite, and what the last page holds behind a sequence is NaN."""
    from oracle_engine_b200.csrc import ops
    lens = [1, 32, 33, 300, 65]
    G, pages = H // KVH, [(n + 63) // 64 for n in lens]
    cache = torch.full((sum(pages) + 1, 2, KVH, 64, hd), float("nan"))
    tables = torch.full((len(lens) + 1, max(pages) + 1), -1, dtype=torch.int32)
    g = torch.Generator().manual_seed(H * 100 + hd)
    order, at = torch.randperm(sum(pages), generator=g).tolist(), 0
    ks, vs = [torch.randn(n, KVH, hd, generator=g) for n in lens], [torch.randn(n, KVH, hd, generator=g) for n in lens]
    for b, n in enumerate(lens):
        if b == 3:
            vs[b][290:] = float("inf")                       # seen by the last ten queries only
        for p in range(pages[b]):
            tables[b, p] = page = order[at]
            at += 1
            m = min(64, n - 64 * p)
            cache[page, 0, :, :m] = ks[b][64 * p:64 * p + m].transpose(0, 1)
            cache[page, 1, :, :m] = vs[b][64 * p:64 * p + m].transpose(0, 1)
    cache, tables = cache.to(dtype).to(DEV), tables.to(DEV)
    rd = lambda t: t.to(dtype).double()                      # noqa: E731
    for mode in ("prompt", "last"):
        seq, pos, rows = [], [], []
        for b, n in enumerate(lens):
            for p in range(n if mode == "prompt" else 1):
                seq.append(b)
                pos.append(p if mode == "prompt" else n - 1 - (15 if b == 3 else 0))
            seq.append(-1)                                   # a padding row between sequences
            pos.append(0)
        T = len(seq)
        q = torch.randn(T, H * hd + 6, generator=g).to(dtype)
        outs = []
        for kind in (0, 1, 2):
            out = torch.full((T, H * hd), 7.0, dtype=dtype, device=DEV)
            ops.attn_paged(out, q.to(DEV), cache, tables, torch.tensor(seq, dtype=torch.int32, device=DEV),
                           torch.tensor(pos, dtype=torch.int32, device=DEV), H, KVH, hd, window, hd ** -0.5, sink, kind)
            outs.append(out.cpu())
        assert torch.equal(outs[0].nan_to_num(9.0, 8.0, -8.0), outs[1].nan_to_num(9.0, 8.0, -8.0))
        assert torch.equal(outs[0].nan_to_num(9.0, 8.0, -8.0), outs[2].nan_to_num(9.0, 8.0, -8.0))
        for t in range(T):
            got = outs[0][t].double().view(H, hd)
            if seq[t] < 0:
                assert (got == 0).all()
                continue
            b, p = seq[t], pos[t]
            if b == 3 and p >= 290:
                continue                                     # infinite values
            lo = max(0, p - window + 1) if window > 0 else p // -window * -window if window < 0 else 0
            for h in (0, H - 1):
                s = (rd(ks[b][lo:p + 1, h // G]) @ rd(q[t, h * hd:(h + 1) * hd])) * hd ** -0.5
                e = torch.exp(s - s.max())
                o = (e @ rd(vs[b][lo:p + 1, h // G])) / (e.sum() + (math.exp(-s.max()) if sink else 0.0))
                assert (got[h] - o).abs().max() <= (2e-5 if dtype == torch.float32 else 2.0 ** -8 * o.abs().max() + 2e-5)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("kind", [1, 2])
@pytest.mark.parametrize("sink", [False, True])
@pytest.mark.parametrize("window", [0, 16])
def test_a_key_of_nan_reaches_the_queries_that_see_it_and_no_others(dtype, kind, sink, window):
    """Keys of NaN: alone in what a query sees of a chunk, beside other keys of their chunk, and in a chunk that is full."""
    from oracle_engine_b200.csrc import ops
    H, KVH, hd, n = 4, 2, 64, 128
    for nans in ((32, 33), (40, 41), (0, 1), (64, 96)):
        cache = _rand(n // 64, 2, KVH, 64, hd, seed=7)
        keys = cache[:, 0].transpose(1, 2).reshape(n, KVH, hd)
        keys[nans[0]:nans[1]] = float("nan")
        cache[:, 0] = keys.view(n // 64, 64, KVH, hd).transpose(1, 2)
        i32 = lambda t: torch.tensor(t, dtype=torch.int32, device=DEV)                       # noqa: E731
        out = torch.full((n, H * hd), 7.0, dtype=dtype, device=DEV)
        ops.attn_paged(out, _rand(n, H * hd, seed=8).to(dtype), cache.to(dtype), i32([[0, 1]]), i32([0] * n), i32(range(n)), H, KVH, hd, window,
                       hd ** -0.5, sink, kind)
        sees = torch.tensor([p >= nans[0] and (window == 0 or nans[1] - 1 > p - window) for p in range(n)])
        got = out.cpu()
        assert torch.isnan(got[sees]).all() and torch.isfinite(got[~sees]).all()


@pytest.mark.parametrize("T,seqs,kind", [(530000, 1, 0), (66000, 66000, 0), (66000, 1, 1)])
def test_attention_of_more_tokens_than_a_grid_s_second_dimension_holds(T, seqs, kind):
    """66,250 tiles of 64 rows, and a CTA per token for 66,000 tokens; the tokens repeat a few."""
    from oracle_engine_b200.csrc import ops
    H, hd = 8, 2
    q, cache = _rand(5, H * hd, seed=9), _rand(1, 2, 1, 64, hd, seed=10)
    tables = torch.zeros(seqs, 1, dtype=torch.int32, device=DEV)
    at = torch.arange(T, device=DEV) % 5
    seq = (torch.arange(T, device=DEV) % seqs).int()
    few, many = torch.empty(5, H * hd, device=DEV), torch.empty(T, H * hd, device=DEV)
    ops.attn_paged(few, q, cache, tables[:1], torch.zeros(5, dtype=torch.int32, device=DEV), torch.arange(5, dtype=torch.int32, device=DEV), H, 1, hd, 0, 1.0)
    ops.attn_paged(many, q[at], cache, tables, seq, at.int(), H, 1, hd, 0, 1.0, False, kind)
    assert torch.equal(many, few[at])
