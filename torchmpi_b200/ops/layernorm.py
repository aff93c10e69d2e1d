"""Layer normalisation with a one-pass backward (csrc/kernels/layernorm.cu).

``LayerNorm(C)`` is an ``nn.LayerNorm`` (autograd function in csrc/bindings/autograd.cpp) over the last dimension whose CUDA path reads each row once
forward and reads ``(x, dy)`` once backward, producing ``dx``, ``dgamma`` and ``dbeta`` together; eager
PyTorch runs the backward as three kernels.  Inputs the kernel does not cover (CPU, widths that are not
a multiple of 256 bf16 / 128 fp32 elements or above 2048 / 1024, parameters of another dtype) take
``F.layer_norm``.
"""
from __future__ import annotations

import torch
import torch.nn as nn
import torch.nn.functional as F

from .. import _native
from .._lib import lib, dtype_code, has_symbol, TorchMPIError


def __getattr__(name: str):
    if name == "launch_count":               # kernels launched by this module
        return _native.launches(_native.LAYERNORM)
    raise AttributeError(f"module {__name__!r} has no attribute {name!r}")


def supported(x: torch.Tensor, weight, bias) -> bool:
    return (x.is_cuda and weight is not None and bias is not None and weight.dtype == x.dtype and bias.dtype == x.dtype
            and x.dtype in (torch.bfloat16, torch.float16, torch.float32) and has_symbol("tmpi_layernorm_fwd")
            and bool(lib.tmpi_layernorm_supported(x.shape[-1], dtype_code(x.dtype))))


def check_status() -> None:
    """Raises if a layer-norm backward on the current device gave up on one of its bounded waits since the last call."""
    st = lib.tmpi_layernorm_status()
    if st:
        raise TorchMPIError(3, f"layer norm: a bounded wait ran out (code {st})")


def layer_norm_fork(x: torch.Tensor, weight: torch.Tensor, bias: torch.Tensor, eps: float):
    """``(layer_norm(x), x)`` for the two branches of a residual block: in backward the gradients of both outputs are summed by
    the layer norm's kernel.  ``x`` must be ``supported``."""
    return _native.ext().layer_norm_fork(x, weight, bias, eps)


class LayerNorm(nn.LayerNorm):
    def forward(self, x: torch.Tensor) -> torch.Tensor:
        if len(self.normalized_shape) == 1 and supported(x, self.weight, self.bias):
            return _native.ext().layer_norm(x, self.weight, self.bias, self.eps)
        return F.layer_norm(x, self.normalized_shape, self.weight, self.bias, self.eps)
