"""Loads the host extension (csrc/host.cpp) and gives it the entry points of libkd_attention.so.

The extension is the call path of the operator: plan cache, allocations, autograd node, kernel calls. It takes the
library's entry points as addresses, so that whatever library ``_capi`` loaded is the one that runs.
"""
from __future__ import annotations

import ctypes
import importlib.machinery
import importlib.util

import torch  # noqa: F401  (the extension links against libtorch)

from . import _capi
from .build import HOST_PATH

_ENTRY_POINTS = ("kd_plan_layout_get", "kd_classify", "kd_attn_fwd", "kd_attn_bwd", "kd_attn_bwd_hadamard", "kd_attn_fwd_f32", "kd_attn_bwd_f32", "kd_hadamard", "kd_metadata_from_tokens",
                 "kd_cocktail_index", "kd_cocktail_scores", "kd_cocktail_grad", "kd_cast",
                 "kd_last_error")

_ext = None


def load():
    global _ext
    if _ext is None:
        lib = _capi.load()
        if not HOST_PATH.exists():
            raise ImportError(f"{HOST_PATH} is missing: build it with `python -m kerneldev_b200.build`. This package has no other call path.")
        loader = importlib.machinery.ExtensionFileLoader("kd_host", str(HOST_PATH))
        spec = importlib.util.spec_from_file_location("kd_host", str(HOST_PATH), loader=loader)
        ext = importlib.util.module_from_spec(spec)
        loader.exec_module(ext)
        ext.bind({name: ctypes.cast(getattr(lib, name), ctypes.c_void_p).value for name in _ENTRY_POINTS})
        _ext = ext
    return _ext
