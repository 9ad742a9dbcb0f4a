"""What a decode step's merge of split keys makes of values that are no numbers."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("far", [4.0, 16.0])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_a_value_that_is_no_number_shows_however_small_its_weight(far, value):
    """A key whose score lies 16 and 256 below the others', in a split of its own: exp(-256) is zero, and zero times infinity
    is no number, as it is where one CTA takes all keys."""
    from oracle_engine_b200.csrc import ops_tc
    H, G, d, n = 4, 2, 128, 300
    g = torch.Generator().manual_seed(1)
    k, v = torch.zeros(5, G, 64, d), torch.randn(5, G, 64, d, generator=g)
    k[0, :, :, 0] = -far
    v[0, :, 7, 3] = value
    q = torch.zeros(1, H, d)
    q[:, :, 0] = far
    i32 = lambda t: torch.tensor(t, dtype=torch.int32, device=DEV)                            # noqa: E731
    outs = []
    for decode in (True, False):                              # five splits and their merge; one CTA
        ctx = SimpleNamespace(cu_q=i32([0, 1]), seq_start=i32([n - 1]), seq_qlen=i32([1]), n_seqs=1, n_tokens=1, max_qlen=1, max_kvlen=n,
                              all_decode=decode)
        out = torch.zeros(1, H * d, dtype=torch.bfloat16, device=DEV)
        ops_tc.attention_split(out, q.bfloat16().reshape(1, -1).to(DEV), k.bfloat16().to(DEV), v.bfloat16().to(DEV), i32([[0, 1, 2, 3, 4]]), ctx,
                               H, G, d, d, 0, 1.0, 0.0)
        outs.append(out.float().reshape(H, d).cpu())
    for out in outs:
        assert not torch.isfinite(out[:, 3]).any() and torch.isfinite(out[:, :3]).all() and torch.isfinite(out[:, 4:]).all()
    assert ((outs[0] - outs[1]).abs()[:, 4:] <= 2.0 ** -7 * (0.1 + outs[1].abs()[:, 4:])).all()
