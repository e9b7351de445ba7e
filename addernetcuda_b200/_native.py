"""The C++ host path of the eager layer calls (csrc/host.cpp), loaded on the first call with a CUDA tensor.

`layer`, `conv`, `layer_with_stats`, `layer_affine`, `affine` and `column` return None for whatever they do not take - anything but
contiguous fp32 CUDA tensors of a geometry the kernels are built for - and callers then go on in Python, which handles
the rest or raises.  They always call the product library; inside a `_lib.tuning()` block they return None.
"""
from __future__ import annotations

import ctypes
import importlib.util
import sys
import warnings

import torch

from . import _lib

_NAMES = ("adder_b200_status_string", "adder_b200_forward", "adder_b200_forward_stat_slices", "adder_b200_forward_with_stats",
          "adder_b200_forward_affine", "adder_b200_affine_forward",
          "adder_b200_backward_input_workspace_bytes", "adder_b200_backward_input_with_workspace",
          "adder_b200_backward_weight_workspace_bytes", "adder_b200_backward_weight", "adder_b200_conv_forward",
          "adder_b200_conv_backward_input_workspace_bytes", "adder_b200_conv_backward_input_with_workspace",
          "adder_b200_conv_backward_weight_workspace_bytes", "adder_b200_conv_backward_weight")
_ENTRIES = ("layer", "conv", "layer_with_stats", "layer_affine", "affine", "column")
_mod = None


def load() -> None:
    """Load the extension (built first if it is missing or was linked with another torch), bind it to the product library and put
    its entry points in place.  Where that fails, callers get None and a warning: the Python layer needs the library alone."""
    global _mod
    if _mod is None:
        mod = _import()
        if mod is None:
            for name in _ENTRIES:
                globals()[name] = _absent
            return
        _mod = mod
        for name in _ENTRIES:
            globals()[name] = getattr(mod, name)
    sync()


def _import():
    from . import build
    if not build.host_usable() and not build.build_host():
        return None
    spec = importlib.util.spec_from_file_location("_adder_host", build.HOST_LIB)
    try:
        mod = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(mod)
    except ImportError as e:
        warnings.warn(f"{build.HOST_LIB.name} does not load ({e}): eager layer calls go through the Python layer")
        return None
    return mod


def _absent(*args):
    return None


def sync() -> None:
    """Follow `_lib`: bound to the product library, or off while another one is active."""
    if _mod is None:
        return
    from . import adder, adder_cuda
    lib = _lib.load()
    addresses = {n: ctypes.cast(getattr(lib, n), ctypes.c_void_p).value for n in _NAMES} if _lib.is_product(lib) else None
    _mod.bind(addresses, adder.__dict__, adder_cuda.__dict__)


def _first_call(name):
    def call(tensor, *args):
        if not (isinstance(tensor, torch.Tensor) and tensor.is_cuda):
            return None
        load()
        return getattr(sys.modules[__name__], name)(tensor, *args)
    return call


layer, conv, layer_with_stats, layer_affine, affine, column = (_first_call(n) for n in _ENTRIES)
