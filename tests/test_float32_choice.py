"""Which kernel takes a 32-bit product (host rule, no device), by the measured sides of each line."""
import pytest

from oracle_engine_b200.csrc import build

ROWS, TILES64, CHAIN, FOUR, EIGHT = 1, 2, 3, 5, 6


@pytest.mark.parametrize("M,N,K,kind", [
    (1, 2048, 2048, ROWS), (32, 16384, 2048, ROWS), (48, 2048, 2048, ROWS), (64, 2048, 8192, ROWS), (64, 3072, 3072, EIGHT), (64, 16384, 2048, TILES64),
    # a single chain: streamed while that is little, else tiles of 128
    (65, 64, 64, ROWS), (1111, 64, 64, ROWS), (468, 64, 512, ROWS), (130, 512, 64, ROWS), (1111, 128, 64, CHAIN), (130, 2048, 64, CHAIN), (1111, 2048, 512, CHAIN),
    (64, 8192, 512, CHAIN),
    # one round of tiles of 64 where eight shares of tiles of 128 are more than one, two where four shares are
    (130, 3072, 2048, TILES64), (192, 3072, 3072, TILES64), (384, 1536, 2048, TILES64), (1111, 512, 1024, TILES64), (160, 6144, 2048, TILES64),
    (200, 3072, 2048, EIGHT), (256, 2048, 2048, EIGHT), (65, 4096, 4096, EIGHT), (300, 3072, 2048, EIGHT), (384, 3072, 2048, EIGHT), (468, 16384, 2048, FOUR),
    (384, 6144, 2048, FOUR)])
def test_the_rule(M, N, K, kind):
    assert build.load("gemm_simple").oe_gemm_simple_f32_kind(M, N, K, 148) == kind
