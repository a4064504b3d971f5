"""RMSNorm: y = x * rsqrt(mean(x^2) + eps) * w, statistics in 32-bit, the weight a
plain multiplier (src/kernels/norm.cu:73-131 of the reference).  The residual add
that the reference does in a launch of its own (src/kernels/add.cu) is folded in:
the residual stream is 32-bit and the norm adds the pending delta on its way."""
from __future__ import annotations

from typing import List, Mapping, Optional

import torch

from ..ops import kernels as K
from ..weights.loader import WeightSpec
from .base import Part, register_part


class FoldedNorm:
    """The output of an RMSNorm that was never materialised: the product in front of the norm
    left ``xw`` = bfloat16(residual * weight) and the per-tile sums of squares ``ssq`` [tiles, T];
    the product behind it multiplies its result by 1/rms per token (parts/linear.py).  A
    consumer that cannot do that calls ``materialize()``, which runs the norm kernel on the
    (already updated) residual."""

    def __init__(self, norm: "RMSNorm", residual: torch.Tensor, xw: torch.Tensor, ssq: torch.Tensor, ctx):
        self.norm, self.residual, self.xw, self.ssq, self.ctx = norm, residual, xw, ssq, ctx
        self.shape = xw.shape
        self.dtype = xw.dtype

    def materialize(self) -> torch.Tensor:
        out = self.ctx.workspace.get("normed", self.shape, self.ctx.dtype)
        K.add_rms_norm(self.residual, None, self.norm.weight, self.norm.eps, out, None)
        return out


class ReadyNorm(FoldedNorm):
    """The rows of an RMSNorm that the kernel in front of it has already written (the residual is up to date too): handed
    on as a block's ``pending``, taken by that norm's ``forward`` as its result; any other norm just runs."""

    def __init__(self, norm: "RMSNorm", residual: torch.Tensor, rows: torch.Tensor, ctx):
        super().__init__(norm, residual, rows, None, ctx)
        self.rows = rows

    def materialize(self) -> torch.Tensor:
        return self.rows


class NormedSum:
    """rms(a) * wa + rms(b) * wb, not formed yet: two parts' outputs side by side, each under a norm of its own.  The
    kernel that adds the sum into the stream can form it on its way (`RMSNorm.add_normed_then`)."""

    def __init__(self, a: torch.Tensor, wa: torch.Tensor, b: torch.Tensor, wb: torch.Tensor, eps: float, ctx):
        self.a, self.wa, self.b, self.wb, self.eps, self.ctx = a, wa, b, wb, eps, ctx

    def materialize(self, into: Optional[torch.Tensor] = None) -> torch.Tensor:
        """The sum as a float32 tensor, or added into ``into``."""
        out = into if into is not None else self.ctx.workspace.get("normed_sum", tuple(self.a.shape), torch.float32)
        K.sandwich_norm(out, self.a, second=(self.b, self.wa, self.wb, self.eps), keep=into is not None)
        return out


class RMSNorm(Part):
    """Parameters: size, eps; ``weight_offset`` (default 0): the multiplier is ``weight_offset + w`` (1 for a
    weight that is stored around zero); ``tensor``: the weight's full name if it is not ``<prefix>.weight``;
    ``scale_tensor``: the full name of one more vector that multiplies the result element by element (a layer scale behind
    a norm on a part's output), taken into the multiplier."""

    foldable = True                      # fold_buffers / size / eps: the products around it can take it in

    def __init__(self, spec, rt):
        super().__init__(spec, rt)
        self.size = int(self.p("size"))
        self.eps = float(self.p("eps"))
        self.weight_offset = float(self.p("weight_offset", 0.0))
        self.tensor = self.p("tensor", None) or self.name("weight")
        self.scale_tensor = self.p("scale_tensor", None)
        self.weight: Optional[torch.Tensor] = None
        self.fold_tag = "fold.0"          # scratch of the folded form; a block gives its norms different tags

    def weight_specs(self) -> List[WeightSpec]:
        out = [WeightSpec(self.tensor, (self.size,), init="zeros" if self.weight_offset else "norm", as_float32=True)]
        if self.scale_tensor is not None:
            out.append(WeightSpec(self.scale_tensor, (self.size,), init="norm", as_float32=True))
        return out

    def bind(self, tensors: Mapping[str, torch.Tensor]) -> None:
        self.weight = self._vector32(tensors[self.tensor])
        if self.weight_offset:
            self.weight = (self.weight + self.weight_offset).contiguous()     # the multiplier, formed once in 32-bit
        if self.scale_tensor is not None:
            self.weight = (self.weight * self._vector32(tensors[self.scale_tensor])).contiguous()

    def add_normed(self, residual: torch.Tensor, delta: torch.Tensor, ctx, copy=None) -> None:
        """residual += norm(delta): the norm sits on a part's output, the sum goes into the 32-bit stream;
        ``copy`` receives the updated rows in its own type."""
        K.norm_add(residual, delta, self.weight, self.eps, copy)

    def add_normed_then(self, residual: torch.Tensor, delta, ctx, following=None) -> Optional[torch.Tensor]:
        """residual += norm(delta), ``delta`` a tensor or a `NormedSum`; with ``following`` (the RMSNorm in front of the
        next part) its rows too, from the same pass over the stream: returned in the engine's type, else None."""
        second, a = None, delta
        if isinstance(delta, NormedSum):
            a, second = delta.a, (delta.b, delta.wa, delta.wb, delta.eps)
        out = None
        if following is not None:
            out = ctx.workspace.get("normed", tuple(residual.shape), ctx.dtype)
        K.sandwich_norm(residual, a, w=self.weight, eps=self.eps, second=second,
                        w_next=following.weight if following is not None else None,
                        eps_next=following.eps if following is not None else 0.0, out=out)
        return out

    def fold_buffers(self, T: int, ctx, tile: int = 128):
        """(xw [T, size] bfloat16, norm weight, ssq [tiles, T] float32) for a product that folds this
        norm into its residual-adding epilogue, in tiles of ``tile`` columns."""
        tiles = -(-self.size // tile)
        xw = ctx.workspace.get(self.fold_tag + ".xw", (T, self.size), torch.bfloat16)
        ssq = ctx.workspace.get(self.fold_tag + ".ssq", (tiles, T), torch.float32)
        return xw, self.weight, ssq

    def forward(self, residual: torch.Tensor, delta, ctx, *, tag: str = "normed",
                row_idx: Optional[torch.Tensor] = None, may_defer: bool = False, out_dtype=None):
        """Adds ``delta`` (a tensor, None, or a FoldedNorm: then the residual is already updated) into
        the residual and returns the normalised rows (in ``out_dtype``; by default the engine's type).  With
        ``may_defer`` a FoldedNorm made for this very norm is handed on as it is, for the consumer's first
        product to finish."""
        if isinstance(delta, ReadyNorm) and delta.norm is self and row_idx is None and (out_dtype or ctx.dtype) == delta.rows.dtype:
            return delta.rows
        if isinstance(delta, FoldedNorm):
            if may_defer and delta.norm is self and row_idx is None and not isinstance(delta, ReadyNorm):
                return delta
            delta = None
        rows = residual.shape[0] if row_idx is None else row_idx.numel()
        out = ctx.workspace.get(tag, (rows, self.size), out_dtype or ctx.dtype)
        K.add_rms_norm(residual, delta, self.weight, self.eps, out, row_idx)
        return out


class LayerNorm(Part):
    """y = (x - mean) / sqrt(var + eps) * weight + bias, var the mean of the squared deviations, in 32-bit.
    Tensors: ``<prefix>`` + ``weight_leaf`` and ``bias_leaf`` (parameters, so that a checkpoint may call them
    as it likes; ``bias_leaf`` None: no bias).  ``forward`` takes ``delta_scale``: the pending delta is added
    as ``delta_scale * delta`` (a block whose parts' outputs enter the stream times a constant)."""

    takes_delta_scale = True

    def __init__(self, spec, rt):
        super().__init__(spec, rt)
        self.size = int(self.p("size"))
        self.eps = float(self.p("eps"))
        self.weight_leaf = self.p("weight_leaf", ".weight")
        self.bias_leaf = self.p("bias_leaf", ".bias")
        self.weight: Optional[torch.Tensor] = None
        self.bias: Optional[torch.Tensor] = None

    def weight_specs(self) -> List[WeightSpec]:
        out = [WeightSpec(self.prefix + self.weight_leaf, (self.size,), init="norm", as_float32=True)]
        if self.bias_leaf is not None:
            out.append(WeightSpec(self.prefix + self.bias_leaf, (self.size,), init="zeros", as_float32=True))
        return out

    def bind(self, tensors: Mapping[str, torch.Tensor]) -> None:
        self.weight = self._vector32(tensors[self.prefix + self.weight_leaf])
        if self.bias_leaf is not None:
            self.bias = self._vector32(tensors[self.prefix + self.bias_leaf])

    def forward(self, residual: torch.Tensor, delta, ctx, *, tag: str = "normed",
                row_idx: Optional[torch.Tensor] = None, delta_scale: float = 1.0):
        if isinstance(delta, FoldedNorm):        # made for another norm: the residual is already updated
            delta = None
        rows = residual.shape[0] if row_idx is None else row_idx.numel()
        out = ctx.workspace.get(tag, (rows, self.size), ctx.dtype)
        K.add_layer_norm(residual, delta, self.weight, self.bias, self.eps, out, row_idx, delta_scale)
        return out


register_part("norm", "rms_norm", RMSNorm)
register_part("norm", "layer_norm", LayerNorm)
