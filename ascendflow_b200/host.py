"""Loads the native host side (`csrc/host_calls.cpp`): the calls' checks and launches in C++, and the
registered torch op.

`calls` is the module. Its functions launch what they accept and say so; what they refuse has not
been enqueued, and the Python front end (`runtime/`) finds out why. Until `connect()` has given
it the kernel library's entry points it refuses everything, so that the first call of a process goes
through the front end, which builds or verifies that library.
"""

from __future__ import annotations

import ctypes as ct
import importlib.machinery
import importlib.util

import torch  # noqa: F401  (its libraries are what the module links against)

from .build import build_host_library


def _load():
    path = build_host_library()
    loader = importlib.machinery.ExtensionFileLoader("_host_calls", str(path))
    module = importlib.util.module_from_spec(importlib.util.spec_from_loader("_host_calls", loader))
    loader.exec_module(module)
    return module


calls = _load()
_fallback = None
_connected = False


def set_fallback(function):
    """The front end's call for what the registered op refuses."""
    global _fallback
    _fallback = function
    calls.configure(0, 0, 0, function)


def connect():
    """Hand the verified kernel library's entry points over, once."""
    global _connected
    if _connected:
        return
    from .build import library_path
    from .runtime.torch import _library

    library = _library(library_path())
    addresses = (ct.cast(getattr(library, name), ct.c_void_p).value for name in (
        "launch_sparse_mla_kept_status", "launch_sparse_mla_topk_indices", "launch_sparse_mla_cache_append_flagged"))
    calls.configure(*addresses, _fallback)
    _connected = True
