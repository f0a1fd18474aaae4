"""``GCNConv`` -- the module the reference exposes as ``graphcuda.GCNConv``
(src/graphcuda/python/gcn.py:36-48) with its autograd function
(src/graphcuda/python/gcn.py:14-34).

Same constructor, same parameter (one tensor ``weights`` of shape in x out,
initialised ``uniform(-s, s)``, ``s = sqrt(2 / (in + out))`` with the same RNG
consumption), same ``forward(X, adjm)``.  Additive keyword arguments: an
optional ``bias`` (absent by default, so ``state_dict()`` keys are unchanged)
and a ``precision`` switch.
"""
from __future__ import annotations

import math
from typing import Optional

import torch
import torch.nn as nn
from torch.nn.parameter import Parameter

from . import _lib
from .adjacency import as_adjacency, native_handle
from .ops import _prec


class _TracedConv(torch.autograd.Function):
    """The layer inside torch.jit.trace: the trace records this call, where the native node would leave it the output as
    fresh, uninitialised memory."""

    @staticmethod
    def forward(ctx, X, weights, bias, handle, relu, prec, fuse):
        Y, _, inter = _lib.host.layer_forward(X, handle, weights, bias, relu, False, prec)
        ctx.save_for_backward(X, weights, Y, inter)
        ctx.call = handle, relu, prec, fuse, bias is not None
        return Y

    @staticmethod
    def backward(ctx, grad_Y):
        X, weights, Y, inter = ctx.saved_tensors
        handle, relu, prec, fuse, has_bias = ctx.call
        need = ctx.needs_input_grad
        return _lib.host.layer_backward(grad_Y, X, handle, weights, relu, Y, inter, need[0], need[1],
                                        has_bias and need[2], prec, fuse) + (None,) * 4


class GCNConvFunction:
    """Y = relu((adjm @ X) @ weights [+ bias]) as one autograd node (csrc/host/layer.cpp).

    Unlike the reference (python/gcn.py:18) the fp32 mask is not materialised:
    the activation itself is saved and the mask re-derived as Y > 0; the
    aggregated features are saved instead of being recomputed (gcn.cu:40)."""

    @staticmethod
    def apply(X, adjm, weights, apply_relu, bias=None, precision=None, fuse=0):
        # fuse: bit 0 = the incoming gradient is already multiplied by this layer's ReLU mask;
        #       bit 1 = X is the ReLU output of the layer below: gate dX by (X > 0) where it is produced
        prec = _prec(precision)
        h = native_handle(as_adjacency(adjm), prec, needs_symmetry=weights.size(1) < weights.size(0))
        Y = _lib.host.conv(X, h, weights, bias, bool(apply_relu), prec, int(fuse))
        return Y if Y is not None else _TracedConv.apply(X, weights, bias, h, bool(apply_relu), prec, int(fuse))


class GCNConv(nn.Module):
    def __init__(self, in_dim: int, out_dim: int, apply_relu: bool = True, *, bias: bool = False,
                 precision: Optional[str] = None):
        super().__init__()
        self.in_dim = in_dim
        self.out_dim = out_dim
        self.apply_relu = apply_relu
        self.precision = precision
        # Set by a container that knows the layer's neighbours (models.GCN): see GCNConvFunction.forward.
        # Only valid when this layer's output feeds exactly one consumer that gates its input gradient.
        self.fuse_relu_backward = 0

        stdv = math.sqrt(2.0 / (in_dim + out_dim))
        self.weights = Parameter(torch.Tensor(in_dim, out_dim))
        self.weights.data.uniform_(-stdv, stdv)
        if bias:
            self.bias = Parameter(torch.zeros(out_dim))
        else:
            self.register_parameter("bias", None)

    def forward(self, X: torch.Tensor, adjm) -> torch.Tensor:
        return GCNConvFunction.apply(X, adjm, self.weights, self.apply_relu, self.bias, self.precision,
                                     self.fuse_relu_backward)
