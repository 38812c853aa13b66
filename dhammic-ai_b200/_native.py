"""Loader of the native host path (csrc/ssd_torch.so): argument checks, allocations and autograd nodes in C++ on top of the
C-ABI library.  There is no fallback: if either is missing, loading raises."""
from __future__ import annotations

import importlib.machinery
import importlib.util
from pathlib import Path

import torch  # noqa: F401  (the extension links against torch's libraries)

from . import _cabi

_ext = None


def load():
    """The extension module (loaded once)."""
    global _ext
    if _ext is None:
        _cabi.load()
        path = Path(__file__).resolve().parent / "csrc" / "ssd_torch.so"
        if not path.exists():
            raise ImportError(f"{path} is missing: build it first (python {path.parent.parent / 'build.py'}); "
                              "there is no fallback implementation")
        loader = importlib.machinery.ExtensionFileLoader("ssd_torch", str(path))
        spec = importlib.util.spec_from_file_location("ssd_torch", str(path), loader=loader)
        ext = importlib.util.module_from_spec(spec)
        loader.exec_module(ext)
        _ext = ext
    return _ext
