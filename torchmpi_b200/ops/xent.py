"""Softmax cross-entropy whose forward also produces the gradient (one kernel, one read of the logits).

``cross_entropy(logits, labels)`` = mean over rows of ``logsumexp(x) - x[label]``.  On CUDA tensors the
forward kernel writes ``(softmax - onehot) / rows`` next to the loss, so backward is a scalar multiply.
The sum over rows is done by the last block in row order: the loss is bit-reproducible.  The autograd function is
csrc/bindings/autograd.cpp.
"""
from __future__ import annotations

import torch

from .. import _native
from .._lib import has_symbol


def __getattr__(name: str):
    if name == "launch_count":               # kernels launched by this module (read by the benchmark)
        return _native.launches(_native.XENT)
    raise AttributeError(f"module {__name__!r} has no attribute {name!r}")


def cross_entropy(logits: torch.Tensor, labels: torch.Tensor, unit_grad: bool = False) -> torch.Tensor:
    """``unit_grad=True`` is a promise that backward starts at this loss (``loss.backward()``, incoming gradient
    1): the stored gradient is then handed on as it is, without a pass that multiplies it by the incoming
    gradient.  A scaled or combined loss must leave it off."""
    if logits.is_cuda:
        if not has_symbol("tmpi_xent_mean_fwd_bwd_ld"):
            raise RuntimeError("torchmpi_b200: native kernel 'tmpi_xent_mean_fwd_bwd_ld' is missing")
        if logits.dim() != 2 or labels.dtype != torch.int64:
            raise ValueError("cross_entropy expects [rows, classes] logits and int64 labels")
        return _native.ext().cross_entropy(logits, labels.contiguous(), unit_grad)
    return torch.nn.functional.cross_entropy(logits.float(), labels)


class CrossEntropyLoss(torch.nn.Module):
    def __init__(self, unit_grad: bool = False):
        super().__init__()
        self.unit_grad = unit_grad

    def forward(self, logits, labels):
        return cross_entropy(logits, labels, self.unit_grad)
