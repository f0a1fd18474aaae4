"""Fused ``log_softmax`` + ``nll_loss`` for the classification tail of the
reference's training script (tests/gcn/graphcuda_impl.py:24,55)."""
from __future__ import annotations

from typing import Optional

import torch

from . import _lib


class _TracedLoss(torch.autograd.Function):
    """The loss inside torch.jit.trace (see gcn._TracedConv)."""

    @staticmethod
    def forward(ctx, logits, labels, row_mask, scale):
        loss, Z, labels, ws, masked = _lib.host.nll_forward(logits, labels, row_mask, scale)
        ctx.save_for_backward(Z, labels, ws)
        ctx.call = masked, scale
        return loss

    @staticmethod
    def backward(ctx, grad_loss):
        return _lib.host.nll_backward(grad_loss, *ctx.saved_tensors, *ctx.call), None, None, None


def log_softmax_nll_loss(logits: torch.Tensor, labels: torch.Tensor, row_mask: Optional[torch.Tensor] = None,
                         scale: Optional[float] = None) -> torch.Tensor:
    """``F.nll_loss(torch.log_softmax(logits, 1)[row_mask], labels[row_mask])`` in one
    kernel per direction.  ``scale`` defaults to 1 / (number of selected rows)
    (reduction='mean'); pass it explicitly to avoid the host read of the mask
    count, or for a different normalisation (e.g. 1 / global rows in the
    row-partitioned model)."""
    if scale is None:
        cnt = int(row_mask.sum().item()) if row_mask is not None else logits.size(0)
        scale = 1.0 / max(cnt, 1)
    loss = _lib.host.nll_loss(logits, labels, row_mask, scale)
    return loss if loss is not None else _TracedLoss.apply(logits, labels, row_mask, scale)


def argmax_accuracy(logits: torch.Tensor, labels: Optional[torch.Tensor] = None, masks=None, *,
                    want_pred: bool = True):
    """The evaluation tail of the reference's script (tests/gcn/graphcuda_impl.py:63-68) in one kernel.

    Returns ``(pred, counts)``: ``pred`` = ``logits.argmax(dim=1)`` (int64; lowest index among equal
    maxima; None when want_pred is False), ``counts`` = int64 tensor ``[n, 2]`` on the device with, per
    row selection, the number of selected rows predicted right and the number selected (None without
    labels).  ``masks``: None (all rows), one bool / uint8 vector, or a sequence of up to 8 of them.
    Nothing is read back to the host: ``counts[:, 0] / counts[:, 1]`` are the accuracies."""
    if masks is not None:
        masks = [masks] if isinstance(masks, torch.Tensor) and masks.dim() == 1 else list(masks)
    return _lib.host.argmax_accuracy(logits, labels, masks, want_pred)
