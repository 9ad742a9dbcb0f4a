"""The kernels that the rule of the 32-bit products names, at the sizes where it changes: the bits of the general kernel."""
import pytest
import torch

from test_gpu_float32_path import DEV, _rand

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(65, 64, 64), (592, 64, 20), (593, 64, 512),          # streamed, and tiles of 128
                                   (128, 18944, 64), (129, 9473, 36),                    # an SM for each tile; more tiles than SMs
                                   (192, 3072, 516), (193, 3072, 516), (1111, 512, 1024), (129, 6144, 520)])
def test_the_chosen_kernel_gives_the_same_bits(M, N, K):
    from oracle_engine_b200.csrc import ops
    a, w, base = _rand(M, K, seed=1), _rand(N, K, seed=2), _rand(M, N, seed=3)
    plain, out = torch.empty(M, N, device=DEV), torch.full((M + 1, N), 7.0, device=DEV)
    ops.gemm_simple(plain, a, w, kind=4)
    for _ in range(3):                                     # right behind one another
        ops.gemm_simple(out[:M], a, w)
    assert torch.equal(out[:M], plain) and (out[M] == 7.0).all()
    acc = base.clone()
    ops.gemm_simple(acc, a, w, accumulate=True)
    assert torch.equal(acc, base + plain)
