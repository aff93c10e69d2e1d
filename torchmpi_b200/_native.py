"""Loads the C++ autograd functions (csrc/bindings/autograd.cpp, built into lib/_autograd.so by ``build``).

The module's undefined ``tmpi_*`` symbols resolve against the native library that ``_lib`` has loaded globally, in either
flavour of it.  A missing or unloadable module raises: the layers have no second implementation of these functions.
"""
from __future__ import annotations

import importlib.machinery
import importlib.util

from . import _lib, build  # noqa: F401  (_lib loads the native library first)

LINEAR, LAYERNORM, ATTENTION, XENT, ATTENTION_BACKWARD, BATCHNORM, CONV, STEM = range(8)      # counters of ``launches``; attention counts calls
_ext = None


def ext():
    """The extension module (loaded on first use)."""
    global _ext
    if _ext is None:
        if not build.bindings_current():
            build.build_bindings()
        loader = importlib.machinery.ExtensionFileLoader("_autograd", str(build.BINDINGS))
        module = importlib.util.module_from_spec(importlib.util.spec_from_loader("_autograd", loader))
        loader.exec_module(module)
        _ext = module
    return _ext


def launches(what: int) -> int:
    """Kernels (for attention: calls, both ways or backward alone) that the C++ functions of one kind have launched in this
    process; 0 before the first use."""
    return _ext.launches(what) if _ext is not None else 0


def takes(*params) -> bool:
    """Whether the C++ functions take a layer with these parameters: they return every gradient to autograd, so not where a flat
    bucket wants it added in place (``parallel.flat_buckets.direct_grad``)."""
    for p in params:
        if getattr(p, "_tmpi_grad_sink", None) is not None:
            return False
    return True
