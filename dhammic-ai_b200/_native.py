"""Loader of the native host path (csrc/ssd_torch.so): argument checks, allocations and autograd nodes in C++ on top of the
C-ABI library.  There is no fallback: if either is missing, loading raises.  :func:`call` is how the package calls it."""
from __future__ import annotations

import importlib.machinery
import importlib.util
import os
from pathlib import Path

import torch
from torch import Tensor

from . import _cabi

_ext = None
check_status = os.environ.get("SSD_B200_CHECK_STATUS", "0") == "1"


def set_check_status(flag: bool) -> None:
    """The status check of both passes (see ``ssd_scan.set_check_status``), now or when the extension is loaded."""
    global check_status
    check_status = bool(flag)
    if _ext is not None:
        _ext.set_check_status(check_status)


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
        ext.set_check_status(check_status)
        _ext = ext
    return _ext


class _Recorded(torch.autograd.Function):
    """A native operator as one Python autograd function: what ``torch.jit.trace`` can record as a call (of the native code itself it
    sees only the allocations of the outputs) and replay on other inputs."""

    @staticmethod
    def forward(ctx, name, *args):
        ctx.set_materialize_grads(False)
        state = torch._C._get_tracing_state()
        torch._C._set_tracing_state(None)
        try:
            args = [a.detach().requires_grad_(a.requires_grad) if isinstance(a, Tensor) else a for a in args]
            with torch.enable_grad():
                out = getattr(load(), name)(*args)
            single = isinstance(out, Tensor)
            ctx.args, ctx.outs = args, (out,) if single else out
            res = tuple(o.detach() for o in ctx.outs)
            ctx.mark_non_differentiable(*[r for r, o in zip(res, ctx.outs) if not o.requires_grad])
            ctx.save_for_backward(res[0])
        finally:
            torch._C._set_tracing_state(state)
        return res[0] if single else res

    @staticmethod
    def backward(ctx, *grads):
        ctx.saved_tensors  # raises where the graph has been freed
        wanted = [i for i, a in enumerate(ctx.args) if isinstance(a, Tensor) and a.requires_grad]
        pairs = [(o, g) for o, g in zip(ctx.outs, grads) if g is not None and o.requires_grad]
        got = [None] * len(ctx.args)
        if pairs:
            outs, gs = zip(*pairs)
            for i, g in zip(wanted, torch.autograd.grad(outs, [ctx.args[i] for i in wanted], gs, retain_graph=True, allow_unused=True)):
                got[i] = g
        return (None, *got)


def call(name: str, *args):
    """The native operator ``name``; inside ``torch.jit.trace`` through a Python autograd function, which the trace records."""
    if torch.jit.is_tracing():
        return _Recorded.apply(name, *args)
    return getattr(load(), name)(*args)
