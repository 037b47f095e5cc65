"""Build libsplat_b200.so (sm_100a only) and SPLAT/splat_host.so in-tree.

    python triton-fun_b200/build.py [--force] [--verbose]

The library is a plain C-ABI shared object (see include/splat_b200.h); it does not link torch.
splat_host is the Python extension module behind the launchers (csrc/host_binding.cpp): it reads torch's
tensors and calls the library, and is compiled against the installed torch.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
REPO_ROOT = os.path.dirname(PKG_DIR)
CSRC = os.path.join(PKG_DIR, "csrc")
INCLUDE = os.path.join(REPO_ROOT, "include")
LIB_PATH = os.path.join(PKG_DIR, "libsplat_b200.so")
HOST_SRC = os.path.join(CSRC, "host_binding.cpp")
HOST_PATH = os.path.join(PKG_DIR, "SPLAT", "splat_host.so")
HOST_BUILT_FOR = HOST_PATH + ".built-for"      # the torch and Python that it was compiled against

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-shared", "-t", "8",
]


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def headers():
    hs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    hs += [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE)]
    return hs


def up_to_date() -> bool:
    if not os.path.exists(LIB_PATH):
        return False
    t = os.path.getmtime(LIB_PATH)
    return all(os.path.getmtime(f) <= t for f in sources() + headers() + [__file__])


def build_host(force: bool = False) -> str:
    import sysconfig

    import torch
    built_for = f"torch {torch.__version__}, Python {sys.version}"
    if not force and os.path.exists(HOST_PATH) and os.path.exists(HOST_BUILT_FOR) and \
            all(os.path.getmtime(f) <= os.path.getmtime(HOST_PATH) for f in (HOST_SRC, __file__)):
        with open(HOST_BUILT_FOR) as f:
            if f.read() == built_for:
                return HOST_PATH
    root = os.path.dirname(torch.__file__)
    nvcc = shutil.which(os.environ.get("NVCC", "nvcc")) or "/usr/local/cuda/bin/nvcc"
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(nvcc)))
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-w",
           "-I" + os.path.join(root, "include"),
           "-I" + os.path.join(root, "include", "torch", "csrc", "api", "include"),
           "-I" + os.path.join(cuda, "include"), "-I" + sysconfig.get_paths()["include"],
           HOST_SRC, "-o", HOST_PATH, "-L" + os.path.join(root, "lib"),
           "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python"]
    print(" ".join(cmd), file=sys.stderr)
    subprocess.run(cmd, check=True)
    with open(HOST_BUILT_FOR, "w") as f:
        f.write(built_for)
    return HOST_PATH


def build(force: bool = False, verbose: bool = False) -> str:
    build_host(force)
    if not force and up_to_date():
        return LIB_PATH
    nvcc = os.environ.get("NVCC", "nvcc")
    cmd = [nvcc, *NVCC_FLAGS, "-I", INCLUDE, "-I", CSRC]
    if verbose:
        cmd += ["-Xptxas", "-v"]
    cmd += ["-o", LIB_PATH, *sources()]
    print(" ".join(cmd), file=sys.stderr)
    subprocess.run(cmd, check=True)
    return LIB_PATH


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(LIB_PATH)
