"""What ops.sample_rows says about tensors that it does not take (before anything is launched)."""
import pytest
import torch


class _OnDevice:
    """A tensor that says it is on the device."""

    def __init__(self, t):
        self.t = t

    is_cuda = True

    def __getattr__(self, name):
        return getattr(self.t, name)


@pytest.mark.parametrize("bad", ["out", "row_slot", "rng_counter"])
@pytest.mark.parametrize("how", ["type", "stride"])
def test_the_tensor_is_named(bad, how):
    from oracle_engine_b200.csrc import ops
    t = {n: torch.zeros(4, dtype=torch.int32) for n in ("out", "row_slot", "rng_counter")}
    t[bad] = torch.zeros(4, dtype=torch.int64) if how == "type" else torch.zeros(8, dtype=torch.int32)[::2]
    on = {n: _OnDevice(v) for n, v in t.items()}
    with pytest.raises(ops.KernelError, match=f"^{bad} must be a contiguous int32 tensor$"):
        ops.sample_rows(_OnDevice(torch.zeros(4, 8)), on["out"], on["row_slot"], 1.0, 0, 1.0, 1.0, 64, _OnDevice(torch.zeros(4, dtype=torch.int64)),
                        on["rng_counter"], None, None)
