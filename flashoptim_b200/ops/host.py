"""Loader of the native host path (``csrc/fo_host.cpp``): the walk over a parameter group that
packs addresses and launches the fused step kernels.

The extension reads tensors through PyTorch's C++ objects, so it is built against the installed
PyTorch (``flashoptim_b200/build.py``); the kernels themselves stay behind the C ABI of
``libflashoptim_b200.so``, whose entry points are handed over as addresses.

Where it was built for another PyTorch or Python and cannot be built (no compiler, no CUDA headers, a
read-only installation), the Python walk over the group launches the same kernels.
"""

from __future__ import annotations

import ctypes
import importlib.machinery
import importlib.util
import warnings
from types import ModuleType
from typing import Optional

from .. import build as _build
from . import native, step

_module: Optional[ModuleType] = None
_unavailable = False


def loaded() -> Optional[ModuleType]:
    """The extension if some step has loaded it already."""
    return _module


def load() -> ModuleType:
    """Load (building first if it is not that of this source, PyTorch and Python) the extension."""
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


def available() -> Optional[ModuleType]:
    """:func:`load`; None, after one warning, where the extension can be neither loaded nor built."""
    global _unavailable
    if _module is not None or _unavailable:
        return _module
    native.load()  # the kernels themselves are not optional
    try:
        return load()
    except Exception as error:
        _unavailable = True
        warnings.warn(
            f"the native host walk ({_build.HOST_PATH.name}) is not available; steps take the slower Python walk, "
            f"about 6 us of host time per tensor, with the same kernels and results: {error}",
            stacklevel=2,
        )
        return None
