"""Builds libsvdq_b200.so (sm_100a only) with nvcc and the operators' host path `_host.so` with g++, in-tree.

    python -m svdquant_kernels_b200.build [--force] [--verbose]
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
LIB_PATH = os.path.join(PKG_DIR, "libsvdq_b200.so")
HOST_PATH = os.path.join(PKG_DIR, "_host.so")
HEADER = os.path.join(os.path.dirname(PKG_DIR), "include", "svdq_b200.h")


def _sources() -> list[str]:
    out = [os.path.join(CSRC, f) for f in sorted(os.listdir(CSRC)) if f.endswith((".cu", ".cuh", ".h"))]
    out.append(HEADER)
    return out


def _host_sources() -> list[str]:
    return [os.path.join(CSRC, "host_ops.cpp"), HEADER]


def _older(target: str, sources: list[str]) -> bool:
    return not os.path.exists(target) or any(os.path.getmtime(s) > os.path.getmtime(target) for s in sources)


def needs_build() -> bool:
    return _older(LIB_PATH, _sources()) or _older(HOST_PATH, _host_sources())


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile what is older than its sources; return the library's path."""
    if force or _older(LIB_PATH, _sources()):
        _build_library(verbose)
    if force or _older(HOST_PATH, _host_sources()):
        _build_host(verbose)
    return LIB_PATH


def _run(cmd: list[str], what: str, verbose: bool) -> None:
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
    if res.returncode != 0:
        raise RuntimeError(f"{cmd[0]} failed building {what}")


def _build_host(verbose: bool) -> None:
    """The CPython extension `_host` (csrc/host_ops.cpp) against this interpreter's torch."""
    import sysconfig

    import torch
    root = os.path.dirname(torch.__file__)
    includes = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
                sysconfig.get_paths()["include"], "/usr/local/cuda/include"]
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *(f"-I{d}" for d in includes), os.path.join(CSRC, "host_ops.cpp"), "-o", HOST_PATH,
           f"-L{PKG_DIR}", "-lsvdq_b200", "-Wl,-rpath,$ORIGIN",
           f"-L{os.path.join(root, 'lib')}", "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda"]
    _run(cmd, "_host.so", verbose)


def _build_library(verbose: bool) -> None:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found: libsvdq_b200.so cannot be built here")
    cmd = [
        nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
        "-shared", "-Xcompiler", "-fPIC", "-cudart", "static",
        "-o", LIB_PATH, os.path.join(CSRC, "lib.cu"),
    ]
    if verbose:
        cmd.insert(1, "-Xptxas")
        cmd.insert(2, "-v")
    _run(cmd, "libsvdq_b200.so", verbose)


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
