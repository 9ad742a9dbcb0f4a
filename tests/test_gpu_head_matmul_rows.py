"""Per-head products of a handful of tokens, bfloat16 in 16-byte pieces."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("T", [1, 7, 8, 9, 17])
@pytest.mark.parametrize("H,N,K", [(1, 1, 8), (3, 17, 64), (16, 192, 128), (5, 128, 200), (2, 33, 72)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_head_matmul_rows(T, H, N, K, out_dtype):
    from oracle_engine_b200.csrc import ops
    g = torch.Generator().manual_seed(T * 100 + K)
    wide = torch.randn(T, H, K + 8, generator=g).bfloat16().to(DEV)
    w = torch.randn(H, N, K, generator=g).bfloat16().to(DEV)
    a = wide[:, :, :K]
    out = torch.full((T, H, N + 3), 7.0, dtype=out_dtype, device=DEV)
    ops.head_matmul(out[:, :, :N], a, w)
    want = torch.einsum("thk,hnk->thn", a.double(), w.double())
    scale = torch.einsum("thk,hnk->thn", a.double().abs(), w.double().abs())
    # a sum of K products, and the rounding of the result
    bound = lambda want, scale: K * 2.0 ** -24 * scale + (2.0 ** -8 * want.abs() if out_dtype == torch.bfloat16 else 0.0)       # noqa: E731
    assert ((out[:, :, :N].double() - want).abs() <= bound(want, scale)).all()
    assert (out[:, :, N:] == 7.0).all()
    # a token's result does not depend on its neighbours
    one = torch.empty(1, H, N, dtype=out_dtype, device=DEV)
    ops.head_matmul(one, a[T - 1:], w)
    assert torch.equal(one[0], out[T - 1, :, :N])
    # rows off a 16-byte boundary go to the kernel of any alignment
    off = torch.empty(T, H, N, dtype=out_dtype, device=DEV)
    ops.head_matmul(off, wide[:, :, 1:K + 1], w)
    shifted = torch.einsum("thk,hnk->thn", wide[:, :, 1:K + 1].double(), w.double())
    scale = torch.einsum("thk,hnk->thn", wide[:, :, 1:K + 1].double().abs(), w.double().abs())
    assert ((off.double() - shifted).abs() <= bound(shifted, scale)).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_as_many_tokens_as_the_blocks_of_sixteen_reach(dtype):
    """32,768 blocks of 16 tokens: beyond what blocks of eight reach, and not refused."""
    from oracle_engine_b200.csrc import ops
    T, K = 32767 * 16 + 1, 8
    few = torch.randn(7, 1, K, generator=torch.Generator().manual_seed(3)).to(dtype).to(DEV)
    w = torch.randn(1, 3, K, generator=torch.Generator().manual_seed(4)).to(dtype).to(DEV)
    at = torch.arange(T, device=DEV) % 7
    out = torch.empty(T, 1, 3, device=DEV)
    ops.head_matmul(out, few[at], w)
    want = torch.einsum("thk,hnk->thn", few.double(), w.double())
    bound = K * 2.0 ** -24 * torch.einsum("thk,hnk->thn", few.double().abs(), w.double().abs())
    assert ((out.double() - want[at]).abs() <= bound[at]).all()
