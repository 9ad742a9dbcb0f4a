"""What the forms of the decode attention whose warps split the keys take of an SM."""
import pytest

pytestmark = pytest.mark.gpu


def _registers(head_dim, shape):
    from oracle_engine_b200.csrc import ops_tc
    return ops_tc._attn_lib(head_dim).oe_attn_decode_warps_registers(shape[0] * 16 + shape[1])


def test_the_form_of_six_warps_leaves_the_products_their_share():
    """At head size 128 its CTA, one an SM, must leave registers for a product's beside it: 192 threads of 240 are 46,080 of the SM's 65,536."""
    regs = _registers(128, (6, 2))
    assert 0 < regs <= 240, regs
    assert _registers(128, (5, 2)) == -1


@pytest.mark.parametrize("head_dim", [32, 64, 128])
def test_the_rule_counts_ctas_that_an_sm_can_hold(head_dim):
    from oracle_engine_b200.csrc import ops_tc
    warps = {(6, 2): 6, (2, 3): 4, (1, 3): 2}              # the last two: a pair of warps for each
    for shape in ops_tc.DECODE_WARPS_FORMS:
        held = ops_tc.decode_warps_per_sm(shape, head_dim)
        if held:
            granules = (_registers(head_dim, shape) + 7) // 8 * 8
            assert held * warps[shape] * 32 * granules <= 65536, (shape, held, granules)
    if head_dim == 128:
        assert [ops_tc.decode_warps_per_sm(f, 128) for f in ops_tc.DECODE_WARPS_FORMS] == [1, 2, 4]
