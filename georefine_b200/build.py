"""Builds libgeorefine_b200.so (host coder + CUDA kernels + C ABI) in-tree for sm_100a with nvcc and, where there is a C
compiler with this Python's headers, _fastcall, the binding of its hot call for this Python (ctypes makes the call without).

    python -m georefine_b200.build [--force] [--verbose]

The library is written to georefine_b200/_build/ and is rebuilt when any source under csrc/ or include/ is
newer than it.  nvcc cross-compiles without a GPU.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
OUT = PKG / "_build" / "libgeorefine_b200.so"
SOURCES = [CSRC / "capi.cu", CSRC / "bcx_host.cpp", CSRC / "bcx_frame.cpp", CSRC / "bxr_build.cpp"]
FASTCALL_SOURCE = CSRC / "fastcall.c"
FASTCALL = PKG / "_build" / ("_fastcall" + sysconfig.get_config_var("EXT_SUFFIX"))     # (named for the interpreter's ABI)
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC",
         "-Xcompiler", "-pthread", "-shared"]


def _inputs():
    return list(CSRC.glob("*")) + list((PKG.parent / "include").glob("*.h"))


def needs_build() -> bool:
    if not OUT.exists():
        return True
    stamp = OUT.stat().st_mtime
    return any(p.stat().st_mtime > stamp for p in _inputs() if p != FASTCALL_SOURCE)


def build(force: bool = False, verbose: bool = False) -> Path:
    if force or needs_build():
        nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
        if not Path(nvcc).exists():
            raise RuntimeError("nvcc not found: the CUDA library cannot be built here and no prebuilt copy is up to date")
        OUT.parent.mkdir(parents=True, exist_ok=True)
        cmd = [nvcc, *FLAGS, *(["-Xptxas", "-v"] if verbose else []), *map(str, SOURCES), "-o", str(OUT)]
        run = subprocess.run(cmd, capture_output=True, text=True)
        if verbose:
            sys.stderr.write(run.stderr)
        if run.returncode:
            raise RuntimeError("nvcc failed:\n" + run.stderr[-4000:])
    build_fastcall(force)
    return OUT


def build_fastcall(force: bool = False) -> bool:
    """The binding of the hot call for this interpreter; False where it cannot be built."""
    if not force and FASTCALL.exists() and FASTCALL.stat().st_mtime >= FASTCALL_SOURCE.stat().st_mtime:
        return True
    compiler = shutil.which("gcc") or shutil.which("cc")
    if compiler is None:
        return False
    fresh = FASTCALL.with_name(f"{FASTCALL.name}.{os.getpid()}")     # (another process may be loading the finished one)
    try:
        FASTCALL.parent.mkdir(parents=True, exist_ok=True)
        run = subprocess.run([compiler, "-O2", "-fPIC", "-shared", "-I", sysconfig.get_paths()["include"], str(FASTCALL_SOURCE), "-o", str(fresh)],
                             capture_output=True, text=True)
        if run.returncode == 0:
            os.replace(fresh, FASTCALL)
        return run.returncode == 0
    except OSError:
        return False


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
