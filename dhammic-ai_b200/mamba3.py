"""Mamba-3 style variant of the scan: data-dependent rotary state angles and the trapezoidal two-term
discretisation.  The reference's block composes it from two scan calls (src/mamba_base_engine.py:137-187):

    gamma = lam * dt                      beta = (1 - lam) * dt * exp(dt * A_head)
    cum   = -cumsum(raw_angles, dim=1)    B_r, C_r = rope(expand(B), cum), rope(expand(C), cum)
    Y = SSD(x * gamma, dt * A_head, B_r, C_r) + SSD(shift(x) * beta, dt * A_head, shift(B_r), C_r) + D * x

The shifted term at position j+1 reaches every later row i with the decay of position j times
``exp(-a[j+1])``, and ``beta[j+1] * exp(-a[j+1]) = (1 - lam[j+1]) * dt[j+1] =: u[j]``; only the row i = j has no
shifted term.  So the same Y is ONE scan with a combined input weight and a diagonal correction:

    w = lam * dt + u          (u[T-1] = 0)           s = <B, C> per group (the rotation preserves it)
    Y = SSD(x * w, dt * A_head, B_r, C_r) + (D - u * s) * x

which halves the scan work and never materialises shift(x) * beta or shift(B_r).  The element-wise steps and
their backward are CUDA kernels of the library (``ssd_b200_m3_prologue_fwd`` / ``_skip_fwd`` / ``_prologue_bwd``);
the scan runs on the scan kernels (one head per group after the per-head rotation).  On the tensor-core path the
scan takes ``w`` and ``D - u * s`` as per-position coefficients (its scaled operator form) and applies them in
its own prologue and epilogue, so ``x * w`` is never written, the skip term costs no pass over y, and the scan's
backward returns the complete ``dx`` together with ``<dX, x>`` and ``<dy, x>``; the fp32 path materialises
``x * w`` and runs the scan in plain operator form.  Unlike
the reference's cached second call (src/kernels/ssd_scan.py:494-500) the decay gradient is the full one of the
expression above; the chain rule on the (b,T,h)-sized tensors (through w, u and a) is one more kernel
(``ssd_b200_m3_chain_bwd``).
"""
from __future__ import annotations

from torch import Tensor

from . import _native, ssd_scan as _op


def ssd_mamba3(x: Tensor, dt: Tensor, A_head: Tensor, B: Tensor, C: Tensor, D: Tensor | None, raw_angles: Tensor,
               lam: Tensor, chunk_size: int) -> Tensor:
    """x (b,T,h,p); dt, lam (b,T,h) fp32; A_head, D (h); B, C (b,T,g,n); raw_angles (b,T,h,n/2).  Returns Y."""
    return _native.call("mamba3", x, dt, A_head, B, C, D, raw_angles, lam, int(chunk_size), _op._FORCE_PATH, _op._SAVE_STATES)
