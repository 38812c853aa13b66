"""In-tree build of the CUDA library (libssd_b200.so) with nvcc for sm_100a, and of the native host path (ssd_torch.so).

The library is a plain C-ABI shared object (see include/ssd_b200.h); ssd_torch.so is the torch extension that checks
arguments, allocates and calls it.  Both are compiled next to their sources so that a checkout carries its own binaries.
Run ``python -m`` on this file or call :func:`build`.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

CSRC = Path(__file__).resolve().parent / "csrc"
LIB = CSRC / "libssd_b200.so"
HOST_LIB = CSRC / "ssd_torch.so"
HEADER = CSRC.parent.parent / "include" / "ssd_b200.h"
SOURCES = ["ssd_b200_api.cu"]
HOST_SOURCE = "ssd_torch.cpp"
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--expt-extended-lambda", "--expt-relaxed-constexpr", "-shared", "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; the SSD library cannot be built")
    return exe


def _newer(sources, target: Path) -> bool:
    return not target.exists() or max(p.stat().st_mtime for p in sources) > target.stat().st_mtime


def is_stale() -> bool:
    return _newer(list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")) + [HEADER], LIB)


def _run(cmd, what: str) -> str:
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"{what} failed:\n" + res.stdout + res.stderr)
    return res.stderr


def _build_host() -> None:
    import torch
    from torch.utils import cpp_extension
    cuda = Path(_nvcc()).resolve().parent.parent
    inc = cpp_extension.include_paths() + [str(cuda / "include"), sysconfig.get_paths()["include"]]
    lib = Path(torch.__file__).resolve().parent / "lib"
    _run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
          "-DTORCH_EXTENSION_NAME=ssd_torch", *[f for d in inc for f in ("-isystem", d)], str(CSRC / HOST_SOURCE), "-o", str(HOST_LIB),
          f"-L{lib}", f"-L{CSRC}", "-Wl,-rpath,$ORIGIN", "-l:libssd_b200.so", "-ltorch_python", "-ltorch", "-ltorch_cpu",
          "-ltorch_cuda", "-lc10", "-lc10_cuda"], "g++")


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile csrc/*.cu into libssd_b200.so and csrc/ssd_torch.cpp into ssd_torch.so (only what is out of date, unless
    forced)."""
    if force or is_stale():
        cmd = [_nvcc(), *NVCC_FLAGS, "-o", str(LIB)] + [str(CSRC / s) for s in SOURCES]
        if verbose:
            cmd[1:1] = ["-Xptxas", "-v"]
        err = _run(cmd, "nvcc")
        if verbose:
            print(err)
    if force or _newer([CSRC / HOST_SOURCE, HEADER], HOST_LIB):
        _build_host()
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
