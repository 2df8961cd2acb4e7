"""Loads the operator's native host path (bob_torch.so, built from csrc/torch_binding.cpp) and binds it to
libbob_sm100.so.  Only the CUDA route needs it, and there is no fallback: a missing module raises."""

from __future__ import annotations

import ctypes
import importlib.util
import threading
from pathlib import Path

from . import _lib

_MODULE_PATH = Path(__file__).resolve().parent / "bob_torch.so"
_BOUND = ("fwd", "bwd1", "bwd2", "workspace_bytes", "read_status", "last_status", "error_string")

_module = None
_lock = threading.Lock()


def load():
    """The native module, bound to the entry points of the one loaded libbob_sm100.so."""
    global _module
    if _module is not None:
        return _module
    with _lock:
        if _module is None:
            lib = _lib.load()
            if not _MODULE_PATH.exists():
                raise _lib.BobSm100Error(
                    f"{_MODULE_PATH} not found: build it with `python -m flashbob_b200.build`; "
                    "the CUDA route has no fallback")
            spec = importlib.util.spec_from_file_location("flashbob_b200.bob_torch", _MODULE_PATH)
            module = importlib.util.module_from_spec(spec)
            spec.loader.exec_module(module)
            module.bind(_lib.BobSm100Error,
                        *(ctypes.cast(getattr(lib, "bob_sm100_" + n), ctypes.c_void_p).value for n in _BOUND))
            _module = module
    return _module
