"""Builds, in-tree, the C-ABI CUDA library (sglang_b200/lib/libsglang_b200.so) and the extension module of the
torch-facing host path (sglang_b200/_host*.so, csrc/host.cpp).

    python -m sglang_b200.build [--force] [-v]

nvcc cross-compiles for sm_100a; no GPU is needed to build.
"""
from __future__ import annotations

import glob
import os
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB_DIR = os.path.join(PKG, "lib")
LIB = os.path.join(LIB_DIR, "libsglang_b200.so")
HOST_SRC = os.path.join(CSRC, "host.cpp")
HOST = os.path.join(PKG, "_host" + sysconfig.get_config_var("EXT_SUFFIX"))

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-shared",
    "--threads", "0",
]


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _headers():
    return glob.glob(os.path.join(PKG, "..", "include", "*.h")) + glob.glob(os.path.join(CSRC, "*.h"))


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build_host(force: bool = False, verbose: bool = False) -> str:
    """The host path links against the torch of the running interpreter (rebuild after changing torch)."""
    if not force and not _stale(HOST, [HOST_SRC] + _headers()):
        return HOST
    import torch

    root = os.path.dirname(torch.__file__)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-w",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           "-I" + os.path.join(root, "include"), "-I" + os.path.join(cuda, "include"),
           "-I" + sysconfig.get_paths()["include"], "-o", HOST, HOST_SRC, "-L" + os.path.join(root, "lib"),
           "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-ldl"]
    if verbose:
        print(" ".join(cmd))
    subprocess.check_call(cmd)
    return HOST


def build(force: bool = False, verbose: bool = False) -> str:
    build_host(force, verbose)
    if not force and not _stale(LIB, sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + _headers()):
        return LIB
    os.makedirs(LIB_DIR, exist_ok=True)
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    cmd = [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-o", LIB] + sources()
    if verbose:
        print(" ".join(cmd))
    subprocess.check_call(cmd)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
