"""Feed-forward `moe_swiglu`: a mixture of experts with an optional shared expert.

    z = Wr h (float32);  the `top` experts with the largest z are chosen, their weights w_e are the softmax over the
    chosen z alone;  E_e(h) = Wdown_e (silu(Wgate_e h) * (Wup_e h));
    y = sum_chosen w_e E_e(h) + sigmoid(Wsg h) * E_shared(h)                   (the second term only with a shared expert)
Variants by parameter: the weights may be each chosen expert's own sigmoid(z_e), not renormalised; the weight may
multiply the expert's input, y = sum_chosen E_e(w_e h) (its gate and up rows are linear in the input, so the kernel
scales those: silu(w_e g) * (w_e u)); the shared expert may be added without a gate; the choice may be by
sigmoid(z_e) + a learned bias per expert while the weights stay the sigmoids; the logits may have a learned bias of
their own, z = Wr h + br; the experts' unit may be clamped and
shifted, g = min(Wgate h, L), u = clamp(Wup h, -L, L), E_e(h) = Wdown_e (g * sigmoid(1.702 g) * (u + 1)).

Choice by groups (`groups`, a variant of both kinds): the experts stand in `count` equal runs, a run's score is its best
expert's, and only experts of the `keep` best runs can be chosen.

Feed-forward `moe_relu2`: experts without a gate, E_e(h) = Wdown_e max(Wup_e h, 0)^2; by default the weights are the
softmax over ALL experts, the chosen ones divided by their sum (+ 1e-20).

How it is computed: the experts stand side by side in two matrices, all gate and up rows (the shared expert's behind the
routed ones) and all down columns; the router and the shared gate are one small float32 product, whose outcome (a weight
per token and expert, zero where it was not chosen, sigmoid(Wsg h) for the shared one) stays on the device, so a step is
the same kernels whatever the routing (and can be captured in a graph).  By the number of a step's tokens:

* few beside the experts (`_stream_pays`, up to 16, bfloat16): the weight-streaming products over the experts that some token
  chose (csrc/moe_sparse.cu);
* from where it pays (`_sorted_pays`, bfloat16): the (token, expert) pairs sorted by expert and the grouped products over
  them, the arithmetic of the chosen experts and what fills their last row tiles; the shared expert over all tokens;
* else, between the two, in float32 and for sizes those do not take: one product with all gate and up matrices, one kernel that applies the
  unit and multiplies each expert's columns by the token's weight, and one product with all down matrices.
"""
from __future__ import annotations

import torch

from ..csrc import ops
from .linear import chain_flags, matmul_act, matmul_nt, output_flags
from .registry import FEED_FORWARDS, Part
from .spec import TensorDecl


STREAM_TOKENS = 16           # the most tokens that the kernels which stream the chosen experts' weights take


def _stream_pays(T: int, top: int, experts: int) -> bool:
    """Whether T tokens choose few enough of the experts for the kernels that stream the chosen ones' weights; they read at a
    lower rate than the products over all experts, and tokens that choose differently leave little to skip.  us a decode step,
    streamed / all experts, 8 experts of which a token has 2, 8 layers: Fovirax, width 2,048, 2 tokens 530 / 601, 4 607 / 620, 6
    696 / 661, 8 778 / 696, 16 959 / 846, width 3,072, 2 851 / 966, 4 974 / 998, 6 1,072 / 1,035, 16 1,482 / 1,332; Mavinex, width 2,048, 2
    534 / 610, 4 634 / 658, 6 695 / 696, 8 703 / 681, 16 925 / 825; Pusunex, 4 732 / 756, 6 790 / 797, 8 810 / 794, 16 972 / 905.
    (Bogupel with random weights, whose tokens all choose alike, 8 494 / 559.)"""
    return T <= STREAM_TOKENS and T * top <= experts


def _sorted_pays(T: int, top: int, experts: int, D: int, ff: int) -> bool:
    """Whether sorting T tokens by expert saves at least a third of the rows that the products over all experts have (a
    token's rows are its experts', and every expert's last tile of 256 rows is half empty on average), and 130 GFLOP, 0.1 ms: the
    four launches more take 60 us a layer on the host, and as much on the device for what is not the products.  ms a prompt
    step, sorted / all experts, 8 layers: width 1,024 (experts of 704), 2,000 tokens (48 GFLOP) 3.60 / 3.46 Fovirax, 3.26 / 3.13 Mavinex;
    2,048 (1,408), 700 (55) 3.64 / 3.35, 3.33 / 3.00, 1,000 (86) 3.84 / 3.88, 3.16 / 3.31, 1,500 (138) 4.92 / 4.93, 3.71 / 4.11; 3,072
    (2,048), 512 (77) 4.03 / 3.87, 3.38 / 3.38, 700 (120) 4.62 / 4.66, 3.62 / 3.97, Pusunex 4.74 / 4.57, 1,000 (188) 5.23 / 5.67,
    4.25 / 4.92, 5.14 / 5.43."""
    saved = T * experts - (T * top + 128 * experts)
    return 3 * saved >= T * experts and 6.0 * saved * D * ff >= 130e9


def _route(rt, h, w_route, experts: int, top: int, has_gate, dense, ctx, weights, bias, groups) -> None:
    """`dense` from h through the router: one launch where the kernel takes the operands, else a product and the routing.
    float32 sums and logits on both ways and both paths."""
    if rt.tensor_cores and ops.moe_router_supported(h, w_route):
        ops.moe_router(h, w_route, experts, top, has_gate, dense, ctx.tok_seq, weights, bias, groups)
        return
    z = rt.buffer("moe.z", h.shape[0], w_route.shape[0], dtype=torch.float32)
    matmul_nt(rt, z, h, w_route)
    ops.moe_route(z, experts, top, has_gate, dense, ctx.tok_seq, weights=weights, bias=bias, groups=groups)


def _groups(raw, experts: int, top: int):
    """(count, keep) of a choice by groups, or None."""
    if not raw:
        return None
    n, keep = int(raw["count"]), int(raw["keep"])
    if n < 1 or experts % n or not 1 <= keep <= n:
        raise ValueError(f"a mixture of experts: {experts} experts do not stand in {n} equal groups of which {keep} stay")
    if top > keep * (experts // n):
        raise ValueError(f"a mixture of experts: {keep} groups of {experts // n} experts cannot give {top}")
    return n, keep


@FEED_FORWARDS.register("moe_swiglu")
class MoESwiGLU(Part):
    graph_safe = True
    mixture = True
    can_overwrite = True
    """params: hidden_size, num_experts, top, expert_size, shared_size (0 or None: no shared expert), router_weights
    ("softmax", the default: the softmax over the chosen logits alone; "sigmoid": each chosen expert's own
    sigmoid(logit), not renormalised), weight_on ("output", the default: y = sum w_e E_e(h); "input": y = sum E_e(w_e h)),
    shared_gate (default True: the shared expert's output times sigmoid(Wsg h); False: added as it is), choice_bias
    (True: a tensor of one value per expert is added to the sigmoids for the choice alone; needs router_weights
    "sigmoid"), router_bias (True: a tensor of one value per expert is part of the logits; not with "sigmoid"), activation ("silu", the default, or "clamped" with `limit`), groups (None, or {"count", "keep"}), tensor_names (optional overrides of
    "expert" (a format with {e}), "router", "router_bias", "shared", "shared_gate", "choice_bias")."""

    def __init__(self, params, prefix, runtime):
        super().__init__(params, prefix, runtime)
        self.D = int(self._need("hidden_size"))
        self.E = int(self._need("num_experts"))
        self.top = int(self._need("top"))
        self.ff = int(self._need("expert_size"))
        self.sff = int(self.params.get("shared_size") or 0)
        self.router_weights = self.params.get("router_weights") or "softmax"
        self.weight_on = self.params.get("weight_on") or "output"
        self.shared_gate = bool(self.params.get("shared_gate", True)) and self.sff > 0
        self.groups = _groups(self.params.get("groups"), self.E, self.top)
        if self.router_weights not in ("softmax", "sigmoid", "softmax_all") or self.weight_on not in ("output", "input"):
            raise ValueError("moe_swiglu: router_weights is softmax, sigmoid or softmax_all, weight_on is output or input")
        self.choice_bias = bool(self.params.get("choice_bias", False))
        self.router_bias = bool(self.params.get("router_bias", False))
        self.activation = self.params.get("activation") or "silu"
        self.limit = float(self.params.get("limit") or 0.0)
        if self.activation not in ("silu", "clamped") or (self.activation == "clamped" and not self.limit > 0):
            raise ValueError("moe_swiglu: activation is silu or clamped (with a positive limit)")
        if self.activation == "clamped" and self.weight_on != "output":
            raise ValueError("moe_swiglu: the clamped unit is not linear in its input; its weight goes on the output")
        if self.choice_bias and self.router_weights != "sigmoid":
            raise ValueError("moe_swiglu: a choice bias is added to sigmoids; router_weights must be sigmoid")
        if self.router_bias and self.router_weights == "sigmoid":
            raise ValueError("moe_swiglu: a bias on the logits goes with weights that are a softmax")
        if not 1 <= self.top <= self.E:
            raise ValueError(f"moe_swiglu: top {self.top} of {self.E} experts")
        if self.E > 1024:
            raise ValueError("moe_swiglu: up to 1,024 experts are supported")
        names = {"expert": "mlp.e{e}.", "router": "mlp.router", "shared": "mlp.shared.", "shared_gate": "mlp.shared.sg",
                 "choice_bias": "mlp.correction", "router_bias": "mlp.router.b",
                 **self.params.get("tensor_names", {})}
        self.names = {k: prefix + v for k, v in names.items()}
        self.F = self.E * self.ff + self.sff
        self.unit = "clamped" if self.activation == "clamped" else "scale_input" if self.weight_on == "input" else "silu"
        self.sparse = (self.rt.dtype == torch.bfloat16 and self.rt.tensor_cores
                       and ops.moe_sparse_supported(self.D, self.F, self.E, self.ff, self.top))
        self.w_route = self.w_gu = self.w_down = self.bias = None

    def _expert_names(self):
        out = [self.names["expert"].format(e=e) for e in range(self.E)]
        return out + ([self.names["shared"]] if self.sff else [])

    def tensors(self):
        out = []
        for i, p in enumerate(self._expert_names()):
            f = self.ff if i < self.E else self.sff
            out += [TensorDecl(p + "gate", (f, self.D)), TensorDecl(p + "up", (f, self.D)),
                    TensorDecl(p + "down", (self.D, f))]
        out.append(TensorDecl(self.names["router"], (self.E, self.D)))
        if self.shared_gate:
            out.append(TensorDecl(self.names["shared_gate"], (1, self.D)))
        if self.choice_bias:
            out.append(TensorDecl(self.names["choice_bias"], (self.E,)))
        if self.router_bias:
            out.append(TensorDecl(self.names["router_bias"], (self.E,)))
        return out

    def load(self, get):
        to = self.rt.to_compute
        ex = self._expert_names()
        self.w_gu = torch.cat([to(get(p + "gate")) for p in ex] + [to(get(p + "up")) for p in ex], 0).contiguous()
        self.w_down = torch.cat([to(get(p + "down")) for p in ex], 1).contiguous()
        route = [to(get(self.names["router"]))] + ([to(get(self.names["shared_gate"]))] if self.shared_gate else [])
        self.w_route = torch.cat(route, 0).contiguous()
        if self.choice_bias:
            self.bias = self.rt.to_f32(get(self.names["choice_bias"]))
        if self.router_bias:
            self.bias = self.rt.to_f32(get(self.names["router_bias"]))

    def weight_bytes(self):
        return sum(t.numel() * t.element_size() for t in (self.w_gu, self.w_down, self.w_route) if t is not None)

    def flops(self, start, count):
        return count * 2.0 * self.D * (3 * self.F + self.w_route_rows())

    def w_route_rows(self):
        return self.E + (1 if self.shared_gate else 0)

    def first_weights(self):
        return self.w_gu

    def forward(self, h, residual, ctx, overwrite: bool = False):
        """overwrite: the output is written into `residual` (float32) instead of added."""
        T = h.shape[0]
        dense = self.rt.buffer("moe.dense", T, self.E + (1 if self.sff else 0), dtype=torch.float32)
        _route(self.rt, h, self.w_route, self.E, self.top, (True if self.shared_gate else "one") if self.sff else False,
               dense, ctx, self.router_weights, self.bias, self.groups)
        aligned = h.stride(1) == 1 and h.stride(0) % 8 == 0 and h.data_ptr() % 16 == 0
        if self.sparse and aligned and _stream_pays(T, self.top, self.E):
            a = self.rt.buffer("moe.a", T, self.F)
            ops.moe_up_stream(a, h, self.w_gu, dense, self.E, self.ff, self.unit, self.limit, self.top)
            ops.moe_down_stream(residual, a, self.w_down, dense, self.E, self.ff, accumulate=not overwrite)
            return
        if self.sparse and aligned and _sorted_pays(T, self.top, self.E, self.D, self.ff):
            self._forward_sorted(h, residual, dense, overwrite)
            return
        gu = self.rt.buffer("moe.gu", T, 2 * self.F)
        matmul_nt(self.rt, gu, h, self.w_gu)
        a = self.rt.buffer("moe.a", T, self.F)
        ops.moe_dense_act(a, gu, dense, self.E, self.ff, scale_input=self.weight_on == "input", act=self.activation,
                          limit=self.limit)
        matmul_nt(self.rt, residual, a, self.w_down, accumulate=not overwrite, early=output_flags(self.w_down))


    def _forward_sorted(self, h, residual, dense, overwrite: bool) -> None:
        from ..csrc import ops_tc
        rt, T, E, ff = self.rt, h.shape[0], self.E, self.ff
        most = ops.moe_max_tiles(T, self.top, E)
        likely = -(-T * self.top // ops.MOE_ROW_TILE) + E // 2
        rows = most * ops.MOE_ROW_TILE
        i32 = torch.int32
        xs, place = rt.buffer("moe.xs", rows, self.D), rt.buffer("moe.place", T, self.top, dtype=i32)
        row_w, tiles = rt.buffer("moe.row_w", rows, dtype=torch.float32), rt.buffer("moe.tiles", most + 1, dtype=i32)
        ops.moe_place(dense, h, E, self.top, xs, place, row_w, tiles, rt.buffer("moe.counts", (T + 7) // 8 * E, dtype=i32))
        a, y = rt.buffer("moe.a", rows, ff), rt.buffer("moe.y", rows, self.D, dtype=torch.float32)
        ops_tc.gemm_grouped(a, xs, self.w_gu, ff, tiles, likely, row_w=row_w, unit=self.unit, limit=self.limit)
        ops_tc.gemm_grouped(y, a, self.w_down, ff, tiles, likely)
        ops.moe_combine(residual, y, place, accumulate=not overwrite)
        if self.sff:
            a = rt.buffer("moe.a", T, self.sff)
            ops_tc.gemm_grouped(a, h, self.w_gu, self.sff, first=E * ff, row_w=dense[:, E], unit=self.unit, limit=self.limit)
            ops_tc.gemm_grouped(residual, a, self.w_down, self.sff, first=E * ff, accumulate=True)


@FEED_FORWARDS.register("moe_relu2")
class MoEReLU2(Part):
    graph_safe = True
    mixture = True
    can_overwrite = True
    """params: hidden_size, num_experts, top, expert_size, groups (None, or {"count", "keep"}), router_weights
    ("softmax_all", the default, "softmax" or "sigmoid", as csrc/ops.py: moe_route), tensor_names (optional overrides of
    "expert" (a format with {e}) and "router")."""

    def __init__(self, params, prefix, runtime):
        super().__init__(params, prefix, runtime)
        self.D = int(self._need("hidden_size"))
        self.E = int(self._need("num_experts"))
        self.top = int(self._need("top"))
        self.ff = int(self._need("expert_size"))
        self.groups = _groups(self.params.get("groups"), self.E, self.top)
        self.router_weights = self.params.get("router_weights") or "softmax_all"
        if not 1 <= self.top <= self.E <= 1024:
            raise ValueError(f"moe_relu2: top {self.top} of {self.E} experts (up to 1,024 are supported)")
        names = {"expert": "mlp.e{e}.", "router": "mlp.router", **self.params.get("tensor_names", {})}
        self.names = {k: prefix + v for k, v in names.items()}
        self.F = self.E * self.ff
        self.w_route = self.w_up = self.w_down = None

    def tensors(self):
        out = []
        for e in range(self.E):
            p = self.names["expert"].format(e=e)
            out += [TensorDecl(p + "up", (self.ff, self.D)), TensorDecl(p + "down", (self.D, self.ff))]
        return out + [TensorDecl(self.names["router"], (self.E, self.D))]

    def load(self, get):
        to = self.rt.to_compute
        ex = [self.names["expert"].format(e=e) for e in range(self.E)]
        self.w_up = torch.cat([to(get(p + "up")) for p in ex], 0).contiguous()
        self.w_down = torch.cat([to(get(p + "down")) for p in ex], 1).contiguous()
        self.w_route = to(get(self.names["router"]))

    def weight_bytes(self):
        return sum(t.numel() * t.element_size() for t in (self.w_up, self.w_down, self.w_route) if t is not None)

    def flops(self, start, count):
        return count * 2.0 * self.D * (2 * self.F + self.E)

    def first_weights(self):
        return self.w_route

    joint_weight = "w_up"

    def joint_epilogue(self, h, ctx):
        """The routing, and what the up product does with its sums: squared ReLU times the token's weight for the
        column's expert (zero where it was not chosen)."""
        T = h.shape[0]
        dense = self.rt.buffer("moe.dense", T, self.E, dtype=torch.float32)
        _route(self.rt, h, self.w_route, self.E, self.top, False, dense, ctx, self.router_weights, None, self.groups)
        return "relu2", (dense, self.ff)

    def forward(self, h, residual, ctx, overwrite: bool = False, projected=None):
        """overwrite: the output is written into `residual` (float32) instead of added.  projected: the weighted,
        activated up product, computed by the caller."""
        T, a = h.shape[0], projected
        if a is None:
            act, weights = self.joint_epilogue(h, ctx)
            a = self.rt.buffer("moe.a", T, self.F)
            matmul_act(self.rt, a, h, self.w_up, act, weights, early=chain_flags("ffn_in", T))
        matmul_nt(self.rt, residual, a, self.w_down, accumulate=not overwrite, early=chain_flags("ffn_out", T),
                  then=self.rt.next_weights)
