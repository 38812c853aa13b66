"""CPU tests of the C-ABI boundary: the library builds and loads, exports every symbol the header
declares, the ctypes structures match the C layout, and host-side validation answers without a GPU."""
import ctypes as C
import re
import subprocess
import sys
from pathlib import Path

import pytest
import torch

ROOT = Path(__file__).resolve().parents[1]
HEADER = ROOT / "include" / "ssd_b200.h"


def declared_functions():
    text = re.sub(r"/\*.*?\*/", "", HEADER.read_text(), flags=re.S)
    return sorted(set(re.findall(r"\b(ssd_b200_[a-z0-9_]+)\s*\(", text)))


def test_header_declares_expected_entry_points(cabi):
    assert set(declared_functions()) == set(cabi.EXPORTS)


def test_library_exports_every_declared_symbol(cabi):
    lib = cabi.load()
    for name in declared_functions():
        assert hasattr(lib, name), name
    assert lib.ssd_b200_abi_version() == cabi.ABI_VERSION


def test_ctypes_structs_match_c_layout(cabi, tmp_path):
    src = tmp_path / "layout.c"
    src.write_text(
        '#include <stdio.h>\n#include <stddef.h>\n#include "ssd_b200.h"\n'
        'int main(void){printf("%zu %zu %zu %zu %zu %zu %zu\\n", sizeof(ssd_b200_shape), sizeof(ssd_b200_fwd_args),'
        'sizeof(ssd_b200_bwd_args), offsetof(ssd_b200_fwd_args, workspace), offsetof(ssd_b200_bwd_args, dinit),'
        'offsetof(ssd_b200_bwd_args, workspace_bytes), offsetof(ssd_b200_fwd_args, a_cumsum));return 0;}\n')
    exe = tmp_path / "layout"
    subprocess.run(["gcc", "-std=c99", "-Wall", "-Werror", "-I", str(ROOT / "include"), str(src), "-o", str(exe)],
                   check=True)
    got = [int(v) for v in subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split()]
    want = [C.sizeof(cabi.Shape), C.sizeof(cabi.FwdArgs), C.sizeof(cabi.BwdArgs), cabi.FwdArgs.workspace.offset,
            cabi.BwdArgs.dinit.offset, cabi.BwdArgs.workspace_bytes.offset, cabi.FwdArgs.a_cumsum.offset]
    assert got == want


def _shape(cabi, **kw):
    base = dict(abi_version=cabi.ABI_VERSION, dtype=cabi.F32, a_dtype=cabi.F32, path=cabi.PATH_SIMT, batch=2,
                seqlen=512, nheads=8, headdim=64, dstate=64, ngroups=1, chunk=64)
    base.update(kw)
    return cabi.Shape(**base)


def test_host_validation_without_gpu(cabi):
    lib = cabi.load()
    s = _shape(cabi)
    assert lib.ssd_b200_resolve_path(C.byref(s)) == cabi.PATH_SIMT
    fwd = lib.ssd_b200_workspace_bytes(C.byref(s), cabi.PASS_FWD)
    bwd = lib.ssd_b200_workspace_bytes(C.byref(s), cabi.PASS_BWD)
    assert fwd >= 2 * 8 * 8 * 64 * 64 * 4 and bwd > 2 * fwd
    bad = _shape(cabi, seqlen=500)
    assert lib.ssd_b200_resolve_path(C.byref(bad)) == cabi.EINVAL
    assert "not divisible by chunk_size" in cabi.last_error()
    with pytest.raises(AssertionError, match="not divisible"):
        cabi.check(cabi.EINVAL)
    assert lib.ssd_b200_workspace_bytes(C.byref(bad), cabi.PASS_FWD) == 0
    assert lib.ssd_b200_resolve_path(C.byref(_shape(cabi, ngroups=3))) == cabi.EINVAL
    assert lib.ssd_b200_resolve_path(C.byref(_shape(cabi, abi_version=99))) == cabi.EINVAL
    assert lib.ssd_b200_resolve_path(C.byref(_shape(cabi, headdim=512))) == cabi.EUNSUPPORTED
    # argument checks happen before any CUDA call
    args = cabi.FwdArgs(shape=s)
    assert lib.ssd_b200_fwd(C.byref(args), None) == cabi.EINVAL
    assert lib.ssd_b200_fwd(None, None) == cabi.EINVAL
    assert lib.ssd_b200_bwd(None, None) == cabi.EINVAL


@pytest.mark.parametrize("T,refused", [(64, True), (192, True), (128, False)])
def test_row_sums_of_squares_need_whole_tiles(cabi, T, refused):
    """`ysq` holds one entry per position of whole 128-position tiles; a sequence that ends inside a tile would be written past
    it.  The call is refused on the host (and where it is not, it ends for want of a GPU, not of a check)."""
    if torch.cuda.is_available():
        pytest.skip("the accepted case would run with pointers that are none")
    lib = cabi.load()
    s = cabi.Shape(cabi.ABI_VERSION, cabi.BF16, cabi.F32, cabi.PATH_TC, 2, T, 2, 64, 128, 1, 64)
    p = 4096
    a = cabi.FwdArgs(s, p, None, p, p, p, p, p, None, p, p, p, 0, 0, p, 1 << 40, None, None, p, None)
    rc = lib.ssd_b200_fwd(C.byref(a), None)
    assert rc < 0 and (rc == cabi.EINVAL and "whole tiles" in cabi.last_error()) == refused


def test_kept_states_take_no_more_room_than_x(cabi):
    """What a forward holds for the backward on the SIMT path: at most x again and one state, nothing where a chunk's state is
    larger than its x."""
    lib = cabi.load()
    for dtype, width in ((cabi.F32, 4), (cabi.BF16, 2)):
        for n in (8, 16, 64, 128, 256):
            for l in (16, 32, 64, 128):
                s = _shape(cabi, dtype=dtype, path=cabi.PATH_SIMT, dstate=n, chunk=l)
                x = s.batch * s.seqlen * s.nheads * s.headdim * width
                got = lib.ssd_b200_states_bytes(C.byref(s))
                assert got <= x + 256 + 4 * s.batch * s.nheads * s.headdim * n
                assert (got > 0) == (n * 4 <= l * width)


def test_operator_rejects_cpu_tensors(pkg, cabi):
    x = torch.zeros(1, 64, 2, 8)
    with pytest.raises(AssertionError):
        pkg.fused_ssd_scan(x, torch.zeros(1, 64, 2), torch.zeros(1, 64, 2, 4), torch.zeros(1, 64, 2, 4), 32)


def test_forward_mode_is_refused(pkg, cabi):
    """A dual tensor ends in an exception in every operator, whichever argument it is (a dropped tangent would read as zero)."""
    import torch.autograd.forward_ad as fwd
    x, dt, h1, B = torch.zeros(1, 64, 2, 8), torch.zeros(1, 64, 2), torch.zeros(2), torch.zeros(1, 64, 1, 8)
    ang, w = torch.zeros(1, 64, 2, 4), torch.ones(16)
    init, cum = torch.zeros(1, 2, 8, 8), torch.zeros(1, 2, 2, 32)
    calls = {
        "mamba2": ([x, dt, h1, B, B, h1, init], lambda a: pkg.ssd_mamba2(*a[:6], 32, a[6])),
        "operator": ([x, dt, B, B, init, cum], lambda a: pkg.fused_ssd_scan(*a[:4], 32, a[4], {"A_cumsum": a[5]})),
        "gated": ([x, dt, h1, B, B, h1, x, w, init], lambda a: pkg.ssd_mamba2_gated(*a[:8], 1e-6, 32, a[8])),
        "mamba3": ([x, dt, h1, B, B, h1, ang, dt], lambda a: pkg.ssd_mamba3(*a, 32)),
        "rope": ([x, ang], lambda a: pkg.fused_rope(*a)),
        "norm": ([x, x, torch.ones(8)], lambda a: pkg.fused_gate_norm(*a)),
        "trapezoid": ([dt, dt, h1, h1], lambda a: pkg.fused_trapezoidal(*a)),
    }
    for name, (args, call) in calls.items():
        for i in range(len(args)):
            with fwd.dual_level(), pytest.raises(NotImplementedError, match="jvp"):
                call([fwd.make_dual(t.clone(), torch.ones_like(t)) if j == i else t for j, t in enumerate(args)])


def test_missing_library_fails_loudly(cabi, monkeypatch, tmp_path):
    monkeypatch.setattr(cabi, "_lib", None)
    monkeypatch.setattr(cabi, "library_path", lambda: tmp_path / "libssd_b200.so")
    with pytest.raises(ImportError, match="no fallback"):
        cabi.load()
