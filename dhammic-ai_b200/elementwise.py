"""The element-wise operators around the scan in the reference's block, with the reference's names, argument
order, checks and dtypes, on CUDA kernels of the library:

* ``FusedRoPE`` / ``fused_rope(x, angles)``                                 (src/kernels/rope.py:228-325)
* ``FusedTrapezoidal`` / ``fused_trapezoidal(dt_raw, lam_raw, dt_bias, A_log)``  (src/kernels/trapezoidal.py:220-335)
* ``FusedRMSNorm`` / ``fused_rmsnorm(x, weight, eps)`` / ``FusedRMSNormModule``  (src/kernels/rmsnorm.py:154-245)
* ``fused_gate_norm(y, z, weight, eps)``: the block's closing ``norm(y) * silu(z)``
  (src/mamba_base_engine.py:189-191) in one pass instead of three

Arithmetic is fp32 inside, results are in the input dtype; there is no CPU path (CPU tensors raise, as in the
reference).  Checks, allocations and autograd nodes are native (csrc/ssd_torch.cpp).
"""
from __future__ import annotations

import torch
from torch import Tensor

from . import _native


class FusedRoPE:
    """Same call signature as the reference's FusedRoPE (src/kernels/rope.py:228-307)."""

    @staticmethod
    def apply(x: Tensor, angles: Tensor) -> Tensor:
        return _native.call("rope", x, angles)


def fused_rope(x: Tensor, angles: Tensor) -> Tensor:
    """Rotation of the interleaved pairs of the last dim of x (B,T,H,D) by angles (B,T,1,D/2) or (B,T,H,D/2);
    same contract as the reference (src/kernels/rope.py:310-325)."""
    return FusedRoPE.apply(x, angles)


class FusedTrapezoidal:
    """Same call signature as the reference's FusedTrapezoidal (src/kernels/trapezoidal.py:220-310)."""

    @staticmethod
    def apply(dt_raw: Tensor, lam_raw: Tensor, dt_bias: Tensor, A_log: Tensor):
        return _native.call("trapezoid", dt_raw, lam_raw, dt_bias, A_log)


def fused_trapezoidal(dt_raw: Tensor, lam_raw: Tensor, dt_bias: Tensor, A_log: Tensor):
    """(dt, dA, beta, gamma), each of dt_raw's shape and dtype; same contract as the reference
    (src/kernels/trapezoidal.py:317-335)."""
    return FusedTrapezoidal.apply(dt_raw, lam_raw, dt_bias, A_log)


class FusedRMSNorm:
    """Same call signature as the reference's FusedRMSNorm (src/kernels/rmsnorm.py:154-219); an optional fourth
    argument z turns it into the gated form ``rmsnorm(x) * silu(z)``."""

    @staticmethod
    def apply(x: Tensor, weight: Tensor, eps: float, *gate: Tensor) -> Tensor:
        return _native.call("rmsnorm", x, weight, float(eps), gate[0] if gate else None)


def fused_rmsnorm(x: Tensor, weight: Tensor, eps: float = 1e-6) -> Tensor:
    """x * rsqrt(mean(x^2) + eps) * weight over the last dim; same contract as the reference
    (src/kernels/rmsnorm.py:222-230)."""
    return FusedRMSNorm.apply(x, weight, eps)


def fused_gate_norm(y: Tensor, z: Tensor, weight: Tensor, eps: float = 1e-6) -> Tensor:
    """rmsnorm(y, weight, eps) * silu(z), the block's step after the scan (src/mamba_base_engine.py:189-191)."""
    return FusedRMSNorm.apply(y, weight, eps, z)


class FusedRMSNormModule(torch.nn.Module):
    """Same interface as the reference's module (src/kernels/rmsnorm.py:232-245)."""

    def __init__(self, d: int, eps: float = 1e-6):
        super().__init__()
        self.weight = torch.nn.Parameter(torch.ones(d))
        self.eps = eps
        self.d = d

    def forward(self, x: Tensor) -> Tensor:
        return fused_rmsnorm(x, self.weight, self.eps)

    def extra_repr(self) -> str:
        return f"d={self.d}, eps={self.eps}"
