"""Which draws of wide rows look for a small top-k's values by a bound (host rule, no device)."""
import pytest

from oracle_engine_b200.csrc import build


@pytest.mark.parametrize("V,smallest,largest", [(128256, 1, 117), (32000, 1, 117), (32769, 1, 33), (65536, 1, 64), (8192, 1, 32), (8193, 1, 33), (131072, 1, 117)])
def test_the_rule(V, smallest, largest):
    """No more tokens than there are warps with values, and no more values at or above the bound (on average) than are worth comparing."""
    rule = build.load("sampling").oe_sample_by_bound
    assert [k for k in range(-1, 300) if rule(k, V)] == list(range(smallest, largest + 1))
