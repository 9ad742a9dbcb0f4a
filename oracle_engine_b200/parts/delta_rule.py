"""Mixer `gated_delta`: a gated delta rule, a recurrent layer whose memory is one matrix S [dk, dv] per
head and sequence.

With h the layer's input, per token:
    q~, k~, v~ = silu(conv(Wq h)), silu(conv(Wk h)), silu(conv(Wv h))   causal convolution over time, per channel
    q = unit(q~) * dk^-1/2,  k = unit(k~)          unit(a) = a / sqrt(|a|^2 + 1e-6), per head
    beta = sigmoid(Wb h),  g = exp(-exp(A_log) * softplus(Wa h + dt_bias))       one per value head
    S <- g S;  u = beta (v - S^T k);  S <- S + k u^T;  o = S^T q
    x += Wo (o / sqrt(mean(o^2) + eps) * w_norm * silu(Wg h))
q and k have kv_heads heads, v has heads heads; value head i reads q/k head i // (heads / kv_heads).

The six projections are one matrix product whose output is float32 (the decays, step sizes and
everything the recurrence reads stay in float32); S and the last taps - 1 projection rows are
per-sequence state (float32).  Prompts, pieces of prompts and single tokens run the same kernels.
"""
from __future__ import annotations

import torch

from ..csrc import ops
from .linear import matmul_nt, output_flags
from .registry import MIXERS, Part
from .spec import StateNeed, TensorDecl

CHUNKS_FROM = 96              # tokens of a step's longest sequence from which its scan goes in chunks
CHUNKS_MAX_TOKENS = 16384     # (the chunks' scratch is 36 KB a token at 16 heads of 128 x 128; in a captured step, which keeps it, at most 27 MB)


def chunked(tokens: int, longest: int, chunks: int, heads: int, dv: int) -> bool:
    """Whether the scan of a step (its padded tokens; the most tokens a sequence brings; the chunks that its sequences make)
    goes in chunks (csrc/delta_chunks.cu) or walks (csrc/recurrent.cu).  In chunks the chain is shorter, but there is more to
    compute, a CTA (16 columns of a head) fills an SM, and a sequence of one token makes a whole chunk: it pays while the
    chunks of all sequences, shared out over 148 SMs, are no more than 1.25 times the longest sequence's.  us, walk / chunks,
    16 heads of 128 x 128: one sequence of 64 26 / 27, 96 38 / 32, 256 98 / 58, 1,111 416 / 256, 4,096 1,525 / 999; 2 of 300
    168 / 145 (not taken), 4 of 300 208 / 305, 8 of 5 10 / 57, 8 of 300 217 / 579, 32 of 40 113 / 472; one of 192 beside 31 of
    1 97 / 271.  8 heads: one of 1,111 415 / 213, 2 of 300 114 / 79, 8 of 300 208 / 306, one of 192 beside 7 of 1 89 / 53,
    beside 31 90 / 133; 24 heads: one of 256 114 / 113 (not taken); 16 of 64 x 64: one of 1,111 300 / 229, 8 of 300 163 / 255."""
    return CHUNKS_FROM <= longest and tokens <= CHUNKS_MAX_TOKENS and heads * (dv // 16) * chunks <= 185 * -(-longest // ops.SCAN_CHUNK)


_NAMES = {"q": "mix.q", "k": "mix.k", "v": "mix.v", "q_conv": "mix.q.conv", "k_conv": "mix.k.conv",
          "v_conv": "mix.v.conv", "b": "mix.b", "a": "mix.a", "A_log": "mix.A_log", "dt_bias": "mix.dt_bias",
          "g": "mix.g", "norm": "mix.norm", "o": "mix.o"}


@MIXERS.register("gated_delta")
class GatedDelta(Part):
    graph_safe = True
    """params: hidden_size, num_heads, num_kv_heads, key_dim, value_dim, conv_taps, eps (of the read-out's
    norm), tensor_names (optional overrides)."""

    def __init__(self, params, prefix, runtime):
        super().__init__(params, prefix, runtime)
        self.D = int(self._need("hidden_size"))
        self.H = int(self._need("num_heads"))
        self.G = int(self._need("num_kv_heads"))
        self.dk = int(self._need("key_dim"))
        self.dv = int(self._need("value_dim"))
        self.taps = int(self._need("conv_taps"))
        self.eps = float(self._need("eps"))
        if self.H % self.G:
            raise ValueError(f"gated_delta: {self.H} heads are not a multiple of {self.G} key heads")
        if not (1 <= self.dk <= 256 and 1 <= self.dv <= 4096 and 1 <= self.taps <= 32):
            raise ValueError("gated_delta: key_dim up to 256, value_dim up to 4096 and 1..32 taps are supported")
        self.C = 2 * self.G * self.dk + self.H * self.dv                    # channels that pass the convolution
        self.P = self.C + self.H * self.dv + 2 * self.H                     # + gate, beta, a
        self.names = {k: prefix + v for k, v in {**_NAMES, **self.params.get("tensor_names", {})}.items()}
        self.w_in = self.w_o = None
        self.one_launch = self.chunks = False          # set with the weights

    def tensors(self):
        n, qk, vv = self.names, self.G * self.dk, self.H * self.dv
        return [TensorDecl(n["q"], (qk, self.D)), TensorDecl(n["k"], (qk, self.D)), TensorDecl(n["v"], (vv, self.D)),
                TensorDecl(n["q_conv"], (qk, self.taps)), TensorDecl(n["k_conv"], (qk, self.taps)),
                TensorDecl(n["v_conv"], (vv, self.taps)), TensorDecl(n["b"], (self.H, self.D)),
                TensorDecl(n["a"], (self.H, self.D)), TensorDecl(n["A_log"], (self.H,)),
                TensorDecl(n["dt_bias"], (self.H,)), TensorDecl(n["g"], (vv, self.D)),
                TensorDecl(n["norm"], (self.dv,), "ones_normal"), TensorDecl(n["o"], (self.D, vv))]

    def load(self, get):
        to, f32, n = self.rt.to_compute, self.rt.to_f32, self.names
        self.w_in = torch.cat([to(get(n[k])) for k in ("q", "k", "v", "g", "b", "a")], 0).contiguous()
        self.conv_w = torch.cat([f32(get(n[k])) for k in ("q_conv", "k_conv", "v_conv")], 0).contiguous()
        self.A_log, self.dt_bias, self.norm_w = f32(get(n["A_log"])), f32(get(n["dt_bias"])), f32(get(n["norm"]))
        self.w_o = to(get(n["o"]))
        # a decode step's mixer in one launch (the 32-bit path keeps the walk whose bits do not depend on how a sequence is cut)
        self.one_launch = (self.rt.dtype == torch.bfloat16 and self.rt.tensor_cores
                           and ops.delta_step_supported(self.G, self.H, self.dk, self.dv, self.taps))

        self.chunks = (self.rt.dtype == torch.bfloat16 and self.rt.tensor_cores
                       and ops.delta_chunks_supported(self.G, self.H, self.dk, self.dv))

    def step_choice(self, step) -> bool:
        return self.chunks and chunked(step.n_tokens, step.longest, step.scan_chunks, self.H, self.dv)

    def state_need(self):
        return {"S": StateNeed((self.H, self.dk, self.dv), torch.float32),
                "conv": StateNeed((max(self.taps - 1, 1), self.C), torch.float32)}

    def weight_bytes(self):
        return sum(t.numel() * t.element_size() for t in (self.w_in, self.w_o) if t is not None)

    def state_bytes_per_query(self) -> int:
        """Bytes of state one sequence's token reads and writes."""
        return 2 * 4 * (self.H * self.dk * self.dv + max(self.taps - 1, 1) * self.C)

    def cache_bytes_per_query(self, context):
        return self.state_bytes_per_query()

    def flops(self, start, count):
        products = 2.0 * self.D * (self.P + self.H * self.dv)
        return count * (products + 6.0 * self.H * self.dk * self.dv)

    def first_weights(self):
        return self.w_in

    can_overwrite = True

    def forward(self, h, residual, ctx, cache, state, owns_cache=True, overwrite: bool = False):
        """overwrite: the output is written into `residual` (float32) instead of added."""
        T, f32 = h.shape[0], torch.float32
        vv = self.H * self.dv
        buf = self.rt.buffer
        proj = buf("delta.proj", T, self.P, dtype=f32)
        matmul_nt(self.rt, proj, h, self.w_in)
        if self.one_launch and ctx.all_decode and ctx.n_tokens == ctx.n_seqs:
            y = buf("delta.y", T, vv)
            ops.delta_step(y, state["S"], state["conv"], proj, self.conv_w, self.A_log, self.dt_bias, self.norm_w, ctx, self.G, self.H,
                           self.dk, self.dv, self.dk ** -0.5, self.eps)
            matmul_nt(self.rt, residual, y, self.w_o, accumulate=not overwrite, early=output_flags(self.w_o))
            return
        qkv = buf("delta.qkv", T, self.C, dtype=f32)
        gb = buf("delta.gb", T, 2 * self.H, dtype=f32)
        ops.short_conv_prepare(qkv, gb, proj, self.conv_w, state["conv"], self.A_log, self.dt_bias, ctx, self.G,
                               self.H, self.dk, self.dv, self.dk ** -0.5)
        ops.conv_state_update(state["conv"], proj, self.C, self.taps, ctx)
        o = buf("delta.o", T, vv, dtype=f32)
        if self.step_choice(ctx):
            blocks = buf("delta.blocks", ops.delta_chunks_floats(ctx, self.H, self.dk, self.dv), dtype=f32)
            ops.delta_chunks(o, state["S"], blocks, qkv, gb, ctx, self.G, self.H, self.dk, self.dv)
        else:
            ops.delta_rule_scan(o, state["S"], qkv, gb, ctx, self.G, self.H, self.dk, self.dv)
        y = buf("delta.y", T, vv)
        ops.head_gate(y, o, proj[:, self.C:self.C + vv], self.norm_w, self.H, self.dv, True, "silu", self.eps)
        matmul_nt(self.rt, residual, y, self.w_o, accumulate=not overwrite, early=output_flags(self.w_o))
