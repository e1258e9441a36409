"""Loader of the native host path (``csrc/fo_host.cpp``): the walk over a parameter group that
packs addresses and launches the fused step kernels.

The extension reads tensors through PyTorch's C++ objects, so it is built against the installed
PyTorch (``flashoptim_b200/build.py``); the kernels themselves stay behind the C ABI of
``libflashoptim_b200.so``, whose entry points are handed over as addresses.
"""

from __future__ import annotations

import ctypes
import importlib.machinery
import importlib.util
from types import ModuleType
from typing import Optional

from .. import build as _build
from . import native, step

_module: Optional[ModuleType] = None


def loaded() -> Optional[ModuleType]:
    """The extension if some step has loaded it already."""
    return _module


def load() -> ModuleType:
    """Load (building first if the source changed and a compiler is present) the extension."""
    global _module
    if _module is not None:
        return _module
    lib = native.load()
    with native._lock:
        if _module is not None:
            return _module
        if not _build.host_is_current():
            _build.build_host()
        loader = importlib.machinery.ExtensionFileLoader("_fo_host", str(_build.HOST_PATH))
        spec = importlib.util.spec_from_file_location("_fo_host", str(_build.HOST_PATH), loader=loader)
        mod = importlib.util.module_from_spec(spec)
        loader.exec_module(mod)
        from ..optim.base import WALKED
        from ..optim.state import MaybeQuantizedTensor

        def address(fn) -> int:
            return ctypes.cast(fn, ctypes.c_void_p).value

        mod.setup(address(lib.fo_adam_step), address(lib.fo_momentum_step), native.chunk_elems(),
                  MaybeQuantizedTensor, step._ensure_status, native.NativeError, step._NVTX, WALKED)
        _module = mod
    return mod
