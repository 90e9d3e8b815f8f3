"""Loader of ``csrc/ff_host.so``, the native host path of the public operators.

The module gets the addresses of the C ABI functions from the libraries ctypes has
loaded (``_lib.py``, ``indexer_logits.py``), so both call into the same instance.  Its
functions return ``None`` for arguments that need the Python layer's full checks.
"""
from __future__ import annotations

import ctypes
import functools
import importlib.util

from . import _lib
from .build import host_module_path

TOPK_FUNCTIONS = ("ff_topk_launch_typed", "ff_topk_launch_handover", "ff_topk_transform_launch", "ff_topk_workspace_bytes")
LOGITS_FUNCTIONS = ("ff_indexer_logits_launch_fresh",)


def _bind(module, lib, names) -> None:
    for name in names:
        module.bind(name, ctypes.cast(getattr(lib, name), ctypes.c_void_p).value)


def _on_error(rc: int, what: str) -> None:
    if what == "indexer_logits_fp8":
        from .indexer_logits import raise_error
        raise_error(rc)
    _lib.check(rc, what)


@functools.lru_cache(maxsize=None)
def load():
    """The module with the top-k library's functions bound; raises if it is missing (there is no fallback)."""
    path = host_module_path()
    if not path.exists():
        raise _lib.LibraryMissingError(f"{path} is missing: build it with `python -m flash_float_jit_kernels_b200.build`")
    import torch  # noqa: F401  (its libraries resolve the module's symbols)
    spec = importlib.util.spec_from_file_location("ff_host", path)
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)
    module.bind("on_error", _on_error)
    _bind(module, _lib.load(), TOPK_FUNCTIONS)
    return module


@functools.lru_cache(maxsize=None)
def topk():
    return load().topk


@functools.lru_cache(maxsize=None)
def transform():
    return load().transform


@functools.lru_cache(maxsize=None)
def scratch():
    return load().scratch


@functools.lru_cache(maxsize=None)
def logits():
    from .indexer_logits import load as load_indexer
    module = load()
    _bind(module, load_indexer(), LOGITS_FUNCTIONS)
    return module.logits
