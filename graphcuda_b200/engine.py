"""Layer-level composition of the kernels: one GCN layer forward, and the
backward form of the reference's entry point.

The composition itself -- the order of the two products, the fused epilogues,
the padded widths, the autograd node -- is native (csrc/host/layer.cpp); this
module gives it the Python signatures the reference-shaped operators and the
partitioned layer use.
"""
from __future__ import annotations

from typing import Optional

import torch

from . import _lib, ops
from .adjacency import native_handle
from .ops import _prec, _require


def _check_layer_args(X, adj, W):
    _require(X.dim() == 2 and W.dim() == 2, "Inputs must be 2D")
    _require(X.is_cuda and W.is_cuda, "Inputs must be CUDA tensors")
    _require(X.dtype == torch.float32 and W.dtype == torch.float32, "Only float32 is supported here")
    _require(adj.shape[1] == X.size(0), "A.cols must match B.rows")
    _require(X.size(1) == W.size(0), "A.cols must match B.rows")


def _padded_width(n_rows: int, in_dim: int, out_dim: int) -> int:
    """Output width a transform-first layer runs on: a multiple of 4 where the problem is large enough."""
    return _lib.host.padded_width(n_rows, in_dim, out_dim)


class _ZeroPadded:
    """The native registry of buffers whose pad columns are known to be zero."""

    def __len__(self) -> int:
        return _lib.host.zero_padded_count()


_zero_padded = _ZeroPadded()


def _pad_cols(t: torch.Tensor, width: int) -> torch.Tensor:
    if t.size(-1) == width:
        return t
    base = _lib.host.zero_padded_base(t, width)
    if base is not None:
        return base
    out = t.new_zeros(t.shape[:-1] + (width,))
    out[..., :t.size(-1)] = t
    return out


def layer_forward(X, adj, W, bias: Optional[torch.Tensor], relu: bool, *, want_mask: bool = False,
                  precision: Optional[str] = None):
    """(Y, mask or None) of relu((A X) W + b)."""
    prec = _prec(precision)
    h = native_handle(adj, prec, needs_symmetry=W.dim() == 2 and W.size(1) < W.size(0))
    Y, mask, _ = _lib.host.layer_forward(X, h, W, bias, relu, want_mask, prec)
    return Y, mask


def layer_backward_reference_form(dY, X, adj, W, relu: bool, mask, *, precision: Optional[str] = None):
    """(dX, dW) from exactly what the reference's backward entry point receives
    (no saved intermediate): src/graphcuda/cuda/gcn.cu:27-52."""
    _check_layer_args(X, adj, W)
    _require(dY.is_cuda and dY.dtype == torch.float32, "Y_grad must be a float32 CUDA tensor")
    prec = _prec(precision)
    h = native_handle(adj, prec, needs_symmetry=False)
    G = ops.mask_mul(dY, mask) if relu else (dY if dY.stride(1) == 1 else dY.contiguous())
    AX = _lib.host.adj_matmul(h, X, prec)
    dW = ops.gemm(AX.t(), G, precision=precision)
    T = ops.gemm(G, W.t(), precision=precision)
    return _lib.host.adj_matmul(h, T, prec), dW
