"""The native host path (csrc/host/bindings.cpp): ops of one GPU without Python between the arguments
and the launch. ``host.gemm``, ``host.rms_norm``, ... return None for anything but the plain case,
and the calling op then takes its general path. The extension is loaded (and built, when its source is
newer and a compiler is there) on first use; there is no Python stand-in for it.
"""
from __future__ import annotations

import ctypes
import importlib.machinery
import importlib.util
import sys
import threading

from . import _build

_lock = threading.Lock()
_FUNCTIONS = ("gemm", "decode", "rms_norm", "bias_rms_norm", "rounded_bias_rms_norm", "all_reduce", "reset")
_NATIVE = ("kr_last_error", "kr_rms_norm", "kr_local_bias_rms_norm", "kr_local_all_reduce", "kr_gemm_scratch", "kr_gemm")


def _load():
    from . import lib as _lib

    with _lock:
        if "gemm" in globals():
            return
        _build.build_host_if_stale()
        path = str(_build.HOST_PATH)
        loader = importlib.machinery.ExtensionFileLoader(_build.HOST_NAME, path)
        spec = importlib.util.spec_from_file_location(_build.HOST_NAME, path, loader=loader)
        mod = importlib.util.module_from_spec(spec)
        loader.exec_module(mod)
        sys.modules[_build.HOST_NAME] = mod
        handle = _lib.lib()
        mod.bind({n: ctypes.cast(getattr(handle, n), ctypes.c_void_p).value for n in _NATIVE}, _lib.KrakenError)
        globals().update({n: getattr(mod, n) for n in _FUNCTIONS})


def reset_if_loaded() -> None:
    if "reset" in globals():
        globals()["reset"]()


def __getattr__(name: str):
    if name not in _FUNCTIONS:
        raise AttributeError(name)
    _load()
    return globals()[name]
