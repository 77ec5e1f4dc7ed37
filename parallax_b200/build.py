"""Build recipe for libplx_sm100.so (hand-written CUDA for sm_100a + the C ABI) and the host side of eager calls in C++
(_plx_host.*.so, against the headers of the installed PyTorch; without it those calls take the slower Python path).

    python -m parallax_b200.build [--force]

Both are built in-tree (``parallax_b200/lib``); nvcc cross-compiles for sm_100a, so no GPU is needed to build.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

from ._paths import CSRC, INCLUDE, LIB_DIR, LIB_PATH, host_path

SOURCES = ["plx_abi.cu", "plx_decode.cu", "plx_train_mma.cu", "plx_fwd_sm100.cu", "plx_bwd_sm100.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-shared",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; cannot build libplx_sm100.so")
    return exe


def _inputs():
    files = [os.path.join(CSRC, f) for f in os.listdir(CSRC)]
    files.append(os.path.join(INCLUDE, "plx_abi.h"))
    return files


def _stale(built: str) -> bool:
    return not os.path.exists(built) or any(os.path.getmtime(f) > os.path.getmtime(built) for f in _inputs())


def is_stale() -> bool:
    return _stale(LIB_PATH) or _stale(host_path())


def _build_host() -> None:
    import sysconfig

    import torch

    inc = os.path.join(os.path.dirname(torch.__file__), "include")
    libs = os.path.join(os.path.dirname(torch.__file__), "lib")
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    dirs = [inc, os.path.join(inc, "torch", "csrc", "api", "include"), sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-Wall",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *[f for d in dirs for f in ("-isystem", d)],
           "-o", host_path(), os.path.join(CSRC, "plx_host.cpp"), f"-L{libs}", f"-L{os.path.join(cuda, 'lib64')}",
           "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", "-lcudart", "-Wl,-z,now"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("g++ failed:\n" + res.stdout + res.stderr)


def _build_library(verbose: bool) -> None:
    cmd = [_nvcc(), *NVCC_FLAGS, *(["-Xptxas", "-v"] if verbose else []), "-o", LIB_PATH,
           *[os.path.join(CSRC, s) for s in SOURCES]]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + res.stdout + res.stderr)
    if verbose:
        print(res.stderr)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile what is missing or older than the sources, the kernels first; returns the path of libplx_sm100.so."""
    os.makedirs(LIB_DIR, exist_ok=True)
    if force or _stale(LIB_PATH):
        _build_library(verbose)
    if force or _stale(host_path()):
        _build_host()
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
