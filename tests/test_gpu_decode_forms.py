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
