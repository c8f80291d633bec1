"""Builds libsspmm_b200.so (nvcc, sm_100a) and the extension module _sspmm_native.so (host compiler) in-tree.

    python -m sspmm_b200.build [--force] [--verbose]
"""
from __future__ import annotations

import os
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB_DIR = os.path.join(PKG, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libsspmm_b200.so")
NATIVE_PATH = os.path.join(LIB_DIR, "_sspmm_native.so")
INCLUDE = os.path.join(os.path.dirname(PKG), "include")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17", "-shared",
    "-Xcompiler", "-fPIC,-fvisibility=default",
]


def _sources(*suffixes):
    out = []
    for root in (CSRC, INCLUDE):
        for f in sorted(os.listdir(root)):
            if f.endswith(suffixes):
                out.append(os.path.join(root, f))
    return out


def is_stale(path: str = LIB_PATH, suffixes=(".cu", ".cuh", ".h")) -> bool:
    if not os.path.exists(path):
        return True
    t = os.path.getmtime(path)
    return any(os.path.getmtime(s) > t for s in _sources(*suffixes))


def _run(cmd, what: str, verbose: bool) -> None:
    if verbose:
        print(" ".join(cmd))
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
    if r.returncode != 0:
        raise RuntimeError(f"{cmd[0]} failed building {what}")


def build_native(verbose: bool = False) -> str:
    import sysconfig

    import torch
    from torch.utils.cpp_extension import include_paths
    libs = os.path.join(os.path.dirname(torch.__file__), "lib")
    inc = include_paths() + [sysconfig.get_paths()["include"], "/usr/local/cuda/include", INCLUDE]
    _run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden", *(f"-I{i}" for i in inc),
          f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", os.path.join(CSRC, "binding.cpp"), "-o", NATIVE_PATH,
          f"-L{libs}", f"-Wl,-rpath,{libs}", f"-L{LIB_DIR}", "-lsspmm_b200", "-Wl,-rpath,$ORIGIN",
          "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda"], "_sspmm_native.so", verbose)
    return NATIVE_PATH


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(LIB_DIR, exist_ok=True)
    if force or is_stale():
        nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
        _run([nvcc, *(["-Xptxas", "-v"] if verbose else []), *NVCC_FLAGS, "-I", INCLUDE, "-o", LIB_PATH, os.path.join(CSRC, "all.cu")],
             "libsspmm_b200.so", verbose)
    if force or is_stale(NATIVE_PATH, (".cpp", ".h")):
        build_native(verbose)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
