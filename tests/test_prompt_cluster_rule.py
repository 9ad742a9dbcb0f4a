"""How many CTAs share a tile's pages in layers with a window or chunks (host rule, no device)."""
import pytest


@pytest.mark.parametrize("window,cluster", [(0, 2), (128, 1), (256, 1), (600, 1), (1024, 2), (2048, 2), (-256, 1), (-1024, 1), (-2048, 2)])
def test_a_tile_that_sees_few_pages_keeps_them(window, cluster):
    from oracle_engine_b200.csrc import ops_tc
    assert ops_tc.prompt_cluster(256, 1, 3, 8, 1, sm_count=148, window=window) == cluster
    assert ops_tc.prompt_cluster(64, 1, 1, 8, 3, sm_count=148, window=window) == (8 if cluster > 1 else 1)
    assert ops_tc.prompt_cluster(256, 1, 3, 8, 0, sm_count=148, window=window) == 1
