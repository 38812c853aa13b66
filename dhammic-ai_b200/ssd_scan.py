"""Host side of the B200 SSD chunked scan: the reference's operator interface over the C ABI.

``FusedSSDScan`` and ``fused_ssd_scan`` keep the names, argument order, return
arity, cache keys and error behaviour of the reference operator
(src/kernels/ssd_scan.py:427-465, :468-533, :539-583) so that the only
production caller (src/mamba_base_engine.py:170-181) runs unchanged.  All
arithmetic happens in the CUDA library behind include/ssd_b200.h, reached through the
native host path (csrc/ssd_torch.cpp: checks, allocations, autograd nodes); PyTorch
only owns device memory and the stream.  There is no CPU or eager fallback:
non-CUDA tensors raise, as in the reference (src/kernels/ssd_scan.py:247).

Differences from the reference, all deliberate:

* ``A`` may be fp32 while x/B/C are bf16; the chunk cumsum, decay factors,
  states and accumulators are always fp32 (the reference keeps them in the
  input dtype).  ``cache["A_cumsum"]`` is therefore fp32.
* ``B``/``C`` may have fewer heads than ``x`` (groups): (b,T,g,n) with g | h.
* ``L`` and ``decay_chunk`` are not needed by these kernels.  The returned
  cache materialises them on first access (same shapes and values as the
  reference, tests/kernels/test_ssd_scan.py:107-110); ``set_eager_cache(True)``
  makes ``FusedSSDScan.apply`` return them eagerly instead of ``None``.
* Backward is a closed form (no re-run under autograd, no host sync such as
  the reference's ``dfinal_state.abs().sum() > 0``, src/kernels/ssd_scan.py:506).
* A cached call returns no gradient for ``A``, exactly like the reference
  (src/kernels/ssd_scan.py:494-500, :533).

``ssd_mamba2`` is the same scan with the caller's input products fused:
Y = SSD(x*dt, dt*A_head, B, C) + D*x with gradients dx, ddt, dA_head, dB, dC, dD.
"""
from __future__ import annotations

import ctypes as C
import os

import torch
from torch import Tensor

from . import _cabi, _native

_EAGER_CACHE = False
_FORCE_PATH = _cabi.PATH_AUTO
_SAVE_STATES = os.environ.get("SSD_B200_SAVE_STATES", "1") == "1"


def set_save_states(flag: bool) -> None:
    """Keep the recurrent states of the forward for the backward (default on) instead of recomputing them in the backward,
    which is what the reference's input-only checkpointing corresponds to (src/kernels/ssd_scan.py:458).  On the tensor-core
    kernels that is one bf16 state per 128 positions (b*T*h*64 elements, the size of x), on the fp32 multiply-adds one fp32 state
    per chunk, and there only where it takes no more room than the chunk's x; the kernels for partial tiles keep none."""
    global _SAVE_STATES
    _SAVE_STATES = bool(flag)


def set_check_status(flag: bool) -> None:
    """After every call, synchronise and raise if a kernel reported a bounded wait that ran out
    (debug / test use: it costs a stream synchronisation per call)."""
    _native.set_check_status(flag)


def _status(lib, shape, ws, dev) -> None:
    if _native.check_status:
        _cabi.check(lib.ssd_b200_device_status(C.byref(shape), _ptr(ws), _stream(dev)))


def set_eager_cache(flag: bool) -> None:
    """Make FusedSSDScan.apply return materialised L / decay_chunk tensors (default: None, lazy)."""
    global _EAGER_CACHE
    _EAGER_CACHE = bool(flag)


def set_kernel_path(path: str) -> None:
    """'auto' (default), 'simt' (fp32 multiply-adds) or 'tc' (tcgen05 kernels; raises if unsupported).  'auto' takes the tcgen05
    kernels for bf16 calls that fill their tiles (headdim 64, d_state 128, whole tiles of 128 positions), runs other bf16 calls
    (headdim above 32 and up to 64, d_state above 32 and up to 128, multiples of 8; any length and chunk) in fp32 arithmetic on
    tensor-core kernels whose operands are cut into bf16 pieces, and the rest on fp32 multiply-adds.  'tc' takes the tcgen05 kernels
    for those others too, which is faster, with the operands of the products rounded to bf16."""
    global _FORCE_PATH
    _FORCE_PATH = {"auto": _cabi.PATH_AUTO, "simt": _cabi.PATH_SIMT, "tc": _cabi.PATH_TC}[path]


def _dt_code(t: Tensor) -> int:
    if t.dtype == torch.float32:
        return _cabi.F32
    if t.dtype == torch.bfloat16:
        return _cabi.BF16
    raise RuntimeError(f"ssd_b200 supports float32 and bfloat16 tensors, got {t.dtype}")


def _ptr(t: Tensor | None):
    return None if t is None else C.c_void_p(t.data_ptr())


def _stream(dev) -> C.c_void_p:
    return C.c_void_p(torch.cuda.current_stream(dev).cuda_stream)


def _make_shape(x: Tensor, a_dtype: int, B: Tensor, chunk: int) -> _cabi.Shape:
    b, T, h, p = x.shape
    return _cabi.Shape(_cabi.ABI_VERSION, _dt_code(x), a_dtype, _FORCE_PATH, b, T, h, p, B.shape[3], B.shape[2],
                       int(chunk))


def _workspace(lib, shape: _cabi.Shape, which: int, dev, summary: bool = False) -> Tensor:
    """The workspace of a call, or the least it runs with: for a summary, and where the device has no room for the whole."""
    least = int(lib.ssd_b200_workspace_min_bytes(C.byref(shape), which))
    nbytes = least if summary else int(lib.ssd_b200_workspace_bytes(C.byref(shape), which))
    if nbytes == 0:
        _cabi.check(lib.ssd_b200_resolve_path(C.byref(shape)))
    try:
        return torch.empty(max(nbytes, 256), dtype=torch.uint8, device=dev)
    except torch.OutOfMemoryError:
        if least >= nbytes:
            raise
    return torch.empty(max(least, 256), dtype=torch.uint8, device=dev)


class LazySSDCache(dict):
    """The operator's cache dict.  ``A_cumsum`` is always present; ``L`` and ``decay_chunk`` are built
    by a small kernel the first time they are read (the production caller only hands the dict back)."""

    def __init__(self, a_cumsum: Tensor, shape, out_dtype: torch.dtype):
        """``shape``: the call's ``_cabi.Shape``, or its fields behind the ABI version as a tuple, which becomes one when needed."""
        super().__init__(A_cumsum=a_cumsum)
        self._shape = shape
        self._dtype = out_dtype

    def _materialize(self, key: str) -> Tensor:
        s = _cabi.Shape(_cabi.ABI_VERSION, *self._shape) if isinstance(self._shape, tuple) else self._shape
        cum = dict.__getitem__(self, "A_cumsum")
        c = s.seqlen // s.chunk
        with torch.cuda.device(cum.device):
            if key == "L":
                out = torch.empty(s.batch, s.nheads, c, s.chunk, s.chunk, dtype=self._dtype, device=cum.device)
                args = (_ptr(out), None)
            else:
                out = torch.empty(s.batch, s.nheads, c + 1, c + 1, dtype=self._dtype, device=cum.device)
                args = (None, _ptr(out))
            lib = _cabi.load()
            _cabi.check(lib.ssd_b200_materialize_cache(C.byref(s), _ptr(cum), args[0], args[1], _dt_code(out),
                                                       _stream(cum.device)))
        dict.__setitem__(self, key, out)
        return out

    def __missing__(self, key):
        if key in ("L", "decay_chunk"):
            return self._materialize(key)
        raise KeyError(key)

    def get(self, key, default=None):
        if key in ("L", "decay_chunk", "A_cumsum"):
            return self[key]
        return dict.get(self, key, default)

    def __contains__(self, key):
        return key in ("L", "decay_chunk", "A_cumsum") or dict.__contains__(self, key)

    def keys(self):
        return ["L", "decay_chunk", "A_cumsum"]

    def peek(self, key):
        """Read an entry without materialising it (None if not built yet)."""
        return dict.get(self, key)


def _run_fwd(x, a, dt, A_head, D, B, Cm, chunk, init4, a_cumsum_in, want_states=False, ysq=None, skip=None, states=None,
             aux_valid=False):
    """Common forward launcher.  Returns (y, final_state fp32 (b,h,p,n), a_cumsum, shape, states or None).
    ``ysq``: optional fp32 buffer (b, T/128, h, 2, 128) for the per-half-row sums of y^2 (tensor-core path).
    ``states``: a buffer to use instead of allocating one; with ``aux_valid`` its per-position arrays were filled by an
    earlier call on the same inputs and are reused."""
    lib = _cabi.load()
    b, T, h, p = x.shape
    n = B.shape[3]
    dev = x.device
    assert T % chunk == 0, f"sequence length {T} not divisible by chunk_size {chunk}"
    a_dtype = _dt_code(a) if a is not None else _cabi.F32
    shape = _make_shape(x, a_dtype, B, chunk)
    with torch.cuda.device(dev):
        y = torch.empty_like(x)
        final = torch.empty(b, h, p, n, dtype=torch.float32, device=dev)
        if a_cumsum_in is not None:
            cum = a_cumsum_in
            if cum.dtype != torch.float32 or not cum.is_contiguous():
                cum = cum.float().contiguous()
            if tuple(cum.shape) != (b, h, T // chunk, chunk):
                raise ValueError(f"A_cumsum cache has shape {tuple(cum.shape)}, expected {(b, h, T // chunk, chunk)}")
        else:
            cum = torch.empty(b, h, T // chunk, chunk, dtype=torch.float32, device=dev)
        ws = _workspace(lib, shape, _cabi.PASS_FWD, dev)
        if states is None and want_states and _SAVE_STATES:
            nbytes = lib.ssd_b200_states_bytes(C.byref(shape))
            if nbytes:
                states = torch.empty(int(nbytes), dtype=torch.uint8, device=dev)
        flags = _cabi.FWD_AUX_VALID if (aux_valid and states is not None) else 0
        args = _cabi.FwdArgs(shape, _ptr(x), _ptr(a), _ptr(dt), _ptr(A_head), _ptr(D), _ptr(B), _ptr(Cm), _ptr(init4),
                             _ptr(y), _ptr(final), _ptr(cum), 1 if a_cumsum_in is not None else 0, flags, _ptr(ws),
                             ws.numel(), _ptr(states), None, _ptr(ysq), _ptr(skip))
        _cabi.check(lib.ssd_b200_fwd(C.byref(args), _stream(dev)))
        _status(lib, shape, ws, dev)
    return y, final, cum, shape, states


class FusedSSDScan:
    """Same call signature as the reference's FusedSSDScan (src/kernels/ssd_scan.py:441-465)."""

    @staticmethod
    def apply(x: Tensor, A: Tensor, B: Tensor, C_: Tensor, chunk_size: int, initial_states: Tensor | None,
              L_cache_in: Tensor | None, decay_chunk_cache_in: Tensor | None, A_cumsum_cache_in: Tensor | None):
        """(Y, final_state, L, decay_chunk, A_cumsum); L and decay_chunk are None unless the eager cache is on."""
        y, final, cum = _native.call("operator_scan", x, A, B, C_, int(chunk_size), initial_states, A_cumsum_cache_in,
                                                     _FORCE_PATH, _SAVE_STATES)
        L = dc = None
        if _EAGER_CACHE:
            lazy = LazySSDCache(cum, _make_shape(x, _cabi.F32, B, int(chunk_size)), x.dtype)
            L = L_cache_in.detach() if L_cache_in is not None else lazy["L"]
            dc = decay_chunk_cache_in.detach() if decay_chunk_cache_in is not None else lazy["decay_chunk"]
        return y, final, L, dc, cum


def fused_ssd_scan(x: Tensor, A: Tensor, B: Tensor, C: Tensor, chunk_size: int,
                   initial_states: Tensor | None = None, cache: dict | None = None):
    """Fused SSD chunked scan; same contract as the reference (src/kernels/ssd_scan.py:539-583).

    x (b,T,h,p); A (b,T,h) log-decay; B, C (b,T,h,n) (or (b,T,g,n)); initial_states (b,1,h,p,n).
    Returns (Y (b,T,h,p), final_state (b,h,p,n), cache {L, decay_chunk, A_cumsum}).
    """
    if cache is not None:
        if isinstance(cache, LazySSDCache):
            L_in, dc_in, ac_in = cache.peek("L"), cache.peek("decay_chunk"), cache.peek("A_cumsum")
        else:
            L_in, dc_in, ac_in = cache.get("L"), cache.get("decay_chunk"), cache.get("A_cumsum")
            if ac_in is None and (L_in is not None or dc_in is not None):
                raise ValueError("a cache must carry A_cumsum; L and decay_chunk alone cannot be reused here")
    else:
        L_in = dc_in = ac_in = None
    Y, final_state, L_out, dc_out, ac_out = FusedSSDScan.apply(
        x, A, B, C, int(chunk_size), initial_states, L_in, dc_in, ac_in)
    # (not the tensors: the cache must not keep them alive; int: while tracing, a size is a tensor)
    dims = tuple(int(v) for v in (*x.shape, B.shape[3], B.shape[2], chunk_size))
    out_cache = LazySSDCache(ac_out, (_dt_code(x), _cabi.F32, _FORCE_PATH, *dims), x.dtype)
    for k, v in (("L", L_out if L_out is not None else L_in), ("decay_chunk", dc_out if dc_out is not None else dc_in)):
        if v is not None:
            dict.__setitem__(out_cache, k, v)
    return Y, final_state, out_cache


def ssd_mamba2(x: Tensor, dt: Tensor, A_head: Tensor, B: Tensor, C: Tensor, D: Tensor | None, chunk_size: int,
               initial_states: Tensor | None = None):
    """Y = SSD(x*dt, dt*A_head, B, C) + D*x, the scan as the caller composes it
    (src/mamba_base_engine.py:170-173, :187 with gamma = dt), in one call.

    x (b,T,h,p) bf16/fp32; dt (b,T,h); A_head (h); B, C (b,T,g,n); D (h) or None;
    initial_states (b,h,p,n) or (b,1,h,p,n).  Returns (Y, final_state fp32 (b,h,p,n)).
    """
    return _native.call("mamba2", x, dt, A_head, B, C, D, int(chunk_size), initial_states, _FORCE_PATH, _SAVE_STATES)


def ssd_mamba2_gated(x: Tensor, dt: Tensor, A_head: Tensor, B: Tensor, C: Tensor, D: Tensor | None, z: Tensor,
                     norm_weight: Tensor, eps: float, chunk_size: int, initial_states: Tensor | None = None):
    """``rmsnorm(Y) * silu(z)`` with ``Y = SSD(x*dt, dt*A_head, B, C) + D*x``: the scan and the block's output stage
    (src/mamba_base_engine.py:170-173, :187, :189-191; norm as src/kernels/rmsnorm.py:75-150) in one operator.

    z has the size of Y ((b,T,h,p) or (b,T,h*p)); norm_weight (h*p,); the norm runs over all heads of a position.
    Returns (out in x's shape, final_state fp32 (b,h,p,n)).  Gradients: x, dt, A_head, B, C, D, z, norm_weight,
    initial_states.
    """
    return _native.call("mamba2_gated", x, dt, A_head, B, C, D, z, norm_weight, float(eps), int(chunk_size), initial_states,
                                       _FORCE_PATH, _SAVE_STATES)


def resolved_path_name(cfg) -> str:
    """'tc' (the tcgen05 kernels) or 'simt' (everything in fp32 arithmetic, on multiply-adds or in bf16 pieces): what the library
    picks for a workload configuration under the current setting."""
    lib = _cabi.load()
    shape = _cabi.Shape(_cabi.ABI_VERSION, _cabi.BF16 if cfg.dtype == "bf16" else _cabi.F32, _cabi.F32, _FORCE_PATH,
                        cfg.batch, cfg.seqlen, cfg.nheads, cfg.headdim, cfg.d_state, cfg.ngroups, cfg.chunk)
    rc = lib.ssd_b200_resolve_path(C.byref(shape))
    _cabi.check(rc)
    return {_cabi.PATH_SIMT: "simt", _cabi.PATH_TC: "tc"}[rc]
