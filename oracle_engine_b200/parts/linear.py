"""out (+)= a @ w.T for the parts: picks the kernel by precision and shape.

bfloat16 goes to the tensor-core kernels (csrc/gemm_tcgen05.cu) where they take the shape;
float32, and shapes those kernels refuse, go to the CUDA-core kernel (csrc/gemm_simple.cu).
The choice depends only on the runtime and on the weight's shape, never on the data.
Role of the reference's projections through `gemm_q` / `gemv_q` / `ops::matmul`
(core/model.cpp:370-381, 537-547).
"""
from __future__ import annotations

import torch

from ..csrc import ops


# How a product for a handful of tokens (the weight-streaming kernel, csrc/gemm_skinny.cu) is
# chained to its neighbours in the stream:
START_EARLY = 1     # it may start, and request its first weights, while the kernel before it drains
TRIGGER_LATE = 2    # the kernel after it may be scheduled only when its CTAs have streamed their weights
# A kernel that starts early behind a long kernel whose trigger comes at its top sits on the SMs
# while that kernel still needs them: START_EARLY belongs behind a short kernel or a TRIGGER_LATE one.
# What consecutive kernels gain by overlapping is a third of a decode step, and which flags give it
# depends on the kernels' forms, so the four products of a block take theirs from this table, found by
# varying one product at a time inside the 28-layer model (3B shape; ms a step at 1 / 8 / 16 sequences:
# 1.60 / 1.71 / 2.11 with these, 2.38 at 16 with the flags of 8 and the tcgen05 kernel for the large weights).
_CHAIN_FLAGS = {
    # product:   up to 8 tokens,               9 to 16 tokens
    "mixer_in":  (START_EARLY,                 START_EARLY),
    "mixer_out": (START_EARLY | TRIGGER_LATE,  TRIGGER_LATE),
    "ffn_in":    (START_EARLY | TRIGGER_LATE,  START_EARLY | TRIGGER_LATE),
    "ffn_out":   (START_EARLY,                 START_EARLY | TRIGGER_LATE),
}


# Products that are given no flags, in the other decoders' longer chains of short kernels, start early and trigger late: behind
# a kernel of any kind they then wait beside it, and nothing starts on the SMs they still stream through (us a decode step
# with none / 1 / 2 / 3 of the flags, one sequence, 8 layers, width 2,048: Fuvipel 487 / 517 / 476 / 460, Fovirax
# 676 / 751 / 661 / 626, Mavinex 619 / 629 / 619 / 611, Pusunex 678 / 689 / 680 / 651, Bogupel 444 / 498 / 430 / 423; at 8 to 16
# sequences mostly 1 to 4 % between none and both).  Goridra has none of them.
DEFAULT_FLAGS = START_EARLY | TRIGGER_LATE


def output_flags(w: torch.Tensor) -> int:
    """Of a product that ends a mixer or feed-forward and is not in the table: as the default, but it starts early only while each
    of its CTAs, of 16 weight rows, can have an SM of 148 to itself.  More of them behind an attention or a scan sat on the SMs
    that the other chains still needed.  us a decode step at width 3,072, none of the flags / the default everywhere / this:
    Bogupel, 1 sequence 588 / 628 / 568, 4 710 / 785 / 645, 16 1,003 / 1,096 / 942; Fovirax, 4 1,043 / 1,069 / 1,003, 8
    1,182 / 1,298 / 1,259, 16 1,744 / 1,550 / 1,485; Fuvipel, 1 600 / 603 / 593; Pusunex, 1 954 / 924 / 930; up to width 2,048 it
    is the default."""
    return DEFAULT_FLAGS if w.shape[0] <= 16 * 148 else TRIGGER_LATE


def chain_flags(product: str, n_tokens: int) -> int:
    """START_EARLY / TRIGGER_LATE for one of a block's four products in a step of n_tokens rows."""
    return _CHAIN_FLAGS[product][0 if n_tokens <= 8 else 1]


def matmul_nt(rt, out: torch.Tensor, a: torch.Tensor, w: torch.Tensor, accumulate: bool = False,
              early: int = DEFAULT_FLAGS, then: torch.Tensor | None = None) -> None:
    """early: START_EARLY and TRIGGER_LATE flags (above); other kernels ignore them.
    then: the weight matrix of the product that runs after this one (a hint, see ops_tc.gemm)."""
    if rt.dtype == torch.bfloat16 and rt.tensor_cores:
        from ..csrc import ops_tc
        scaled = isinstance(a, ops_tc.ScaledRows)
        if scaled or ops_tc.gemm_supported(a, w, out):
            leave = rt.leave_normed(out) if accumulate and rt.leaving else None
            if leave is not None:           # what comes next is a product with many CTAs, not a norm
                early |= TRIGGER_LATE
            ops_tc.gemm(out, a, w, accumulate=accumulate, early=int(early), then=then, leave=leave)
            return
    ops.gemm_simple(out, a, w, accumulate=accumulate)


def matmul_act(rt, out: torch.Tensor, a: torch.Tensor, w: torch.Tensor, act: str, group_weights: tuple | None = None,
               early: int = DEFAULT_FLAGS) -> None:
    """out = act(a @ w.T), act "gelu" or "relu2", out of the compute dtype; with group_weights (float32 [T, groups], ff;
    "relu2" only) column c times weights[:, c // ff].  Where a tensor-core product takes the shapes the activation is its
    epilogue, on the float32 sums; else it is a kernel of its own."""
    if rt.dtype == torch.bfloat16 and rt.tensor_cores:
        from ..csrc import ops_tc
        if ops_tc.gemm_supported(a, w, out):
            ops_tc.gemm(out, a, w, act=act, group_weights=group_weights, early=int(early))
            return
    ops.gemm_simple(out, a, w)
    if group_weights is not None:
        if act != "relu2":
            raise ValueError("group weights go with squared-ReLU experts")
        ops.moe_dense_relu2(out, *group_weights)
    else:
        {"gelu": ops.gelu_, "relu2": ops.relu2_}[act](out)
