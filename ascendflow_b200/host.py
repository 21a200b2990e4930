"""Loads the native host side (`csrc/host_calls.cpp`): the calls' checks and launches in C++, and the
registered torch op.

`calls` is the module. Its functions launch what they accept and say so; what they refuse has not
been enqueued, and the Python front end (`runtime/`) finds out why. Until `connect()` has given
it the kernel library's entry points it refuses everything, so that the first call of a process goes
through the front end, which builds or verifies that library.

Where the module cannot be had (a torch without CUDA, no compiler) the package still imports and traces:
a stand-in refuses everything, and `connect()`, on the way of every call with CUDA tensors, says why.
"""

from __future__ import annotations

import ctypes as ct
import importlib.machinery
import importlib.util

import torch  # noqa: F401  (its libraries are what the module links against)

from .build import build_host_library
from .diagnostics import CompileError


def _load():
    path = build_host_library()
    loader = importlib.machinery.ExtensionFileLoader("_host_calls", str(path))
    module = importlib.util.module_from_spec(importlib.util.spec_from_loader("_host_calls", loader))
    loader.exec_module(module)
    return module


class _Unavailable:
    """Refuses every call; registers the op for tracing, with calls that go through the front end."""

    def __init__(self, error):
        self.error = error

    def configure(self, attention, select, append, fallback):
        if not hasattr(self, "registration"):
            self.registration = torch.library.Library("ascendflow_b200", "DEF")
            self.registration.define(SCHEMA, tags=(torch.Tag.pt2_compliant_tag,))
            self.registration.impl("sparse_mla", fallback, "CUDA")

    def sparse_mla(self, *tensors):
        return False

    def topk_indices(self, *arguments):
        return None

    def cache_append(self, *arguments):
        return None

    def read_status(self):
        raise RuntimeError("the native host side is not available") from self.error

    def release_workspaces(self):
        pass


SCHEMA = ("sparse_mla(Tensor q, Tensor ori_kv, Tensor cmp_kv, Tensor cmp_sparse_indices, Tensor ori_block_table, "
          "Tensor cmp_block_table, Tensor cu_seqlens_q, Tensor seqused_ori_kv, Tensor seqused_cmp_kv, "
          "Tensor cmp_residual_kv, Tensor ori_topk_length, Tensor sinks, Tensor(a12!) attention_out) -> ()")

try:
    calls = _load()
except (CompileError, ImportError, OSError) as error:
    calls = _Unavailable(error)
_fallback = None
_connected = False


def set_fallback(function):
    """The front end's call for what the registered op refuses."""
    global _fallback, _connected
    _fallback = function
    calls.configure(0, 0, 0, function)
    _connected = False  # the neighbouring steps may have handed the entry points over before this was imported


def connect():
    """Hand the verified kernel library's entry points over, once; true when they were not there before."""
    global _connected
    if _connected:
        return False
    if isinstance(calls, _Unavailable):
        raise RuntimeError("the native host side is not available") from calls.error
    from .build import library_path
    from .runtime.torch import _library

    library = _library(library_path())
    addresses = (ct.cast(getattr(library, name), ct.c_void_p).value for name in (
        "launch_sparse_mla_kept_status", "launch_sparse_mla_topk_indices", "launch_sparse_mla_cache_append_flagged"))
    calls.configure(*addresses, _fallback)
    _connected = True
    return True
