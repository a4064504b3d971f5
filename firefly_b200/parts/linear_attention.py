"""Linear attention: with a constant decay per head (`LinearAttention`, the lightning-attention form), and with a decay
per key channel and token (`GatedLinearAttention`, below).  The first:

    q, k = silu(W_q x), silu(W_k x)   [heads, dim];   v = silu(W_v x)   [heads, vdim]
    S_t  = decay_h S_(t-1) + k_t v_t^T;   o_t = S_t^T q_t             per head, S starts at 0
    out  = W_o (rms_norm(o over all heads together) * norm * sigmoid(W_g x))

There is no softmax, no scale and no position encoding.  The request's state slot holds S of every head in
32-bit (in the recurrence kernel's own order); a portion of a prompt continues from it, so prompts may be cut
anywhere.  The four projections are one product against the stacked matrix [q | k | v | g]; the SiLU of q, k, v
is taken in 32-bit where the recurrence reads them (``csrc/ssm.cu``).

Parameters: hidden_size, heads, dim, vdim, decay (one number per head), eps (of the output norm).
Tensors (leaves under the prefix): q, k [heads*dim, W]; v, g [heads*vdim, W]; norm [heads*vdim]; o [W, heads*vdim].
"""
from __future__ import annotations

from typing import List, Mapping

import torch

from ..cache.spec import StateSpec
from ..ops import kernels as K
from ..weights.arena import FusedSpec, Piece
from ..weights.loader import WeightSpec
from .base import Part, register_part
from .linear import apply_linear, scaled_linear_into_residual


class LinearAttention(Part):
    adds_into_residual = True        # forward(accumulate_into=...)
    scales_residual = True           # forward(residual_scale=...)

    def __init__(self, spec, rt, position=None):
        super().__init__(spec, rt)
        self.hidden = int(self.p("hidden_size"))
        self.heads = int(self.p("heads"))
        self.dim = int(self.p("dim"))
        self.vdim = int(self.p("vdim", self.dim))
        self.eps = float(self.p("eps"))
        self.decay_values = tuple(float(a) for a in self.p("decay"))
        if len(self.decay_values) != self.heads:
            raise ValueError(f"{self.prefix}: {len(self.decay_values)} decays for {self.heads} heads")
        self.state_floats = K.scan_state_floats(self.heads, self.dim, self.vdim)
        self.kq, self.kv = self.heads * self.dim, self.heads * self.vdim
        self.w_qkvg = self.w_o = self.norm = self.decay = None

    def cache_spec(self):
        return StateSpec((self.state_floats,), torch.float32)

    def _sources(self):
        return [(self.name("q"), self.kq), (self.name("k"), self.kq), (self.name("v"), self.kv), (self.name("g"), self.kv)]

    def weight_specs(self) -> List[WeightSpec]:
        out = [WeightSpec(name, (rows, self.hidden)) for name, rows in self._sources()]
        out += [WeightSpec(self.name("norm"), (self.kv,), init="norm", as_float32=True),
                WeightSpec(self.name("o"), (self.hidden, self.kv))]
        return out

    def fused_layout(self, dtype_of) -> List[FusedSpec]:
        pieces, at = [], 0
        for name, rows in self._sources():
            pieces.append(Piece(name, at))
            at += rows
        return [FusedSpec(self.name("qkvg"), (at, self.hidden), tuple(pieces))]

    def bind(self, tensors: Mapping[str, torch.Tensor]) -> None:
        if self.name("qkvg") in tensors:
            self.w_qkvg = self._matrix(tensors[self.name("qkvg")])
        else:
            mats = [self._matrix(tensors[name]) for name, _ in self._sources()]
            if len({m.dtype for m in mats}) != 1:
                mats = [m.to(torch.float32) for m in mats]
            self.w_qkvg = torch.cat(mats, dim=0).contiguous()
        self.w_o = self._matrix(tensors[self.name("o")])
        self.norm = self._vector32(tensors[self.name("norm")])
        self.decay = torch.tensor(self.decay_values, dtype=torch.float32, device=self.w_o.device)

    def forward(self, x, ctx, slot: int, write_cache: bool, accumulate_into=None, residual_scale: float = 1.0):
        T, ws = x.shape[0], ctx.workspace
        dt = self.w_qkvg.dtype
        if x.dtype != dt:
            raise K.KernelError(f"{self.prefix}: activations {x.dtype} against matrices {dt}")
        proj = ws.get("lin_attn.proj", (T, 2 * self.kq + 2 * self.kv), dt)
        apply_linear(x, self.w_qkvg, proj, ctx, "lin_attn.proj")
        o = ws.get("lin_attn.o", (T, self.kv), torch.float32)
        K.scalar_decay_scan((proj, 0), (proj, self.kq), (proj, 2 * self.kq), ctx.state(slot), 0, ctx, o, self.heads,
                            self.dim, self.vdim, silu_inputs=True, decay=self.decay)
        y = ws.get("lin_attn.y", (T, self.kv), dt)
        K.gated_rms_norm(o, (proj, 2 * self.kq + self.kv), self.norm, self.eps, y, 1, gate_first=False)
        return scaled_linear_into_residual(y, self.w_o, accumulate_into, residual_scale, ctx, "lin_attn.out")


class GatedLinearAttention(Part):
    """Linear attention with a decay per key channel and token (the gated-linear-attention form):

        q = W_q x * dim^-0.5,  k = W_k x   [heads, dim];   v = W_v x   [heads, vdim]
        z = W_a2 (W_a1 x) + b;   alpha = sigmoid(z)^(1 / tau)          [heads, dim]
        S_t = diag(alpha_t) S_(t-1) + k_t v_t^T;   o_t = S_t^T q_t     per head, S starts at 0
        out = W_o (rms_norm(o over each head) * norm * silu(W_g x))

    q, k, v, the gate and the decay's first projection are one product; the decays are formed in 32-bit by one kernel
    from the low-rank row, the scan is the one of `LinearAttention` with the decays as rows.

    Parameters: hidden_size, heads, dim, vdim, decay_rank, tau, eps (of the heads' norm).
    Tensors: q, k [heads*dim, W]; v, g [heads*vdim, W]; a1 [rank, W]; a2 [heads*dim, rank]; a2.b [heads*dim];
    norm [vdim]; o [W, heads*vdim]."""

    adds_into_residual = True        # forward(accumulate_into=...)
    scales_residual = True           # forward(residual_scale=...)

    def __init__(self, spec, rt, position=None):
        super().__init__(spec, rt)
        self.hidden = int(self.p("hidden_size"))
        self.heads, self.dim = int(self.p("heads")), int(self.p("dim"))
        self.vdim = int(self.p("vdim", self.dim))
        self.rank = int(self.p("decay_rank"))
        self.tau = float(self.p("tau"))
        self.eps = float(self.p("eps"))
        if self.rank <= 0 or not (self.tau > 0):
            raise ValueError(f"{self.prefix}: decay_rank {self.rank} and tau {self.tau} must be positive")
        self.state_floats = K.scan_state_floats(self.heads, self.dim, self.vdim)
        self.kq, self.kv = self.heads * self.dim, self.heads * self.vdim
        self.w_in = self.w_a2 = self.b_a2 = self.w_o = self.norm = None

    def cache_spec(self):
        return StateSpec((self.state_floats,), torch.float32)

    def step_scratch_bytes(self, tokens: int, sequences: int) -> int:
        return K.scan_scratch_bytes(self.rt.dtype, tokens, sequences, self.heads, 1, self.dim, self.vdim, channel_decay=True)

    def _sources(self):
        n = self.name
        return [(n("q"), self.kq), (n("k"), self.kq), (n("v"), self.kv), (n("g"), self.kv), (n("a1"), self.rank)]

    def weight_specs(self) -> List[WeightSpec]:
        n = self.name
        out = [WeightSpec(name, (rows, self.hidden)) for name, rows in self._sources()]
        out += [WeightSpec(n("a2"), (self.kq, self.rank)), WeightSpec(n("a2.b"), (self.kq,), init="zeros", as_float32=True),
                WeightSpec(n("norm"), (self.vdim,), init="norm", as_float32=True), WeightSpec(n("o"), (self.hidden, self.kv))]
        return out

    def fused_layout(self, dtype_of) -> List[FusedSpec]:
        pieces, at = [], 0
        for name, rows in self._sources():
            pieces.append(Piece(name, at))
            at += rows
        return [FusedSpec(self.name("qkvga"), (at, self.hidden), tuple(pieces))]

    def bind(self, tensors: Mapping[str, torch.Tensor]) -> None:
        n = self.name
        if n("qkvga") in tensors:
            self.w_in = self._matrix(tensors[n("qkvga")])
        else:
            mats = [self._matrix(tensors[name]) for name, _ in self._sources()]
            if len({m.dtype for m in mats}) != 1:
                mats = [m.to(torch.float32) for m in mats]
            self.w_in = torch.cat(mats, dim=0).contiguous()
        self.w_a2 = self._matrix(tensors[n("a2")])
        if self.w_a2.dtype != self.w_in.dtype:
            self.w_in, self.w_a2 = self.w_in.to(torch.float32), self.w_a2.to(torch.float32)
        self.w_o = self._matrix(tensors[n("o")])
        self.b_a2, self.norm = self._vector32(tensors[n("a2.b")]), self._vector32(tensors[n("norm")])

    def forward(self, x, ctx, slot: int, write_cache: bool, accumulate_into=None, residual_scale: float = 1.0):
        T, ws, kq, kv = x.shape[0], ctx.workspace, self.kq, self.kv
        dt = self.w_in.dtype
        if x.dtype != dt:
            raise K.KernelError(f"{self.prefix}: activations {x.dtype} against matrices {dt}")
        proj = ws.get("gla.proj", (T, 2 * kq + 2 * kv + self.rank), dt)
        apply_linear(x, self.w_in, proj, ctx, "gla.proj")
        alpha = ws.get("gla.alpha", (T, kq), torch.float32)
        K.low_rank_decay((proj, 2 * kq + 2 * kv), self.w_a2, self.b_a2, self.tau, alpha)
        o = ws.get("gla.o", (T, kv), torch.float32)
        K.scalar_decay_scan((proj, 0), (proj, kq), (proj, 2 * kq), ctx.state(slot), 0, ctx, o, self.heads, self.dim,
                            self.vdim, channel_decay=(alpha, 0), q_scale=float(self.dim) ** -0.5)
        y = ws.get("gla.y", (T, kv), dt)
        K.head_norm_gate(o, (proj, 2 * kq + kv), self.norm, self.eps, y, self.heads, self.vdim, "silu")
        return scaled_linear_into_residual(y, self.w_o, accumulate_into, residual_scale, ctx, "gla.out")


register_part("mixer", "linear_attention", LinearAttention)
register_part("mixer", "gated_linear_attention", GatedLinearAttention)
