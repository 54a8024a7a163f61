"""Builds libsmla_b200.so (the C-ABI CUDA library, nvcc for sm_100a) and _smla_native.so (the CPython extension that holds
the host side of the ops, g++ against torch's headers) in-tree.

    python -m sparse_mla_sm120_b200.build [--force]
"""
from __future__ import annotations

import glob
import os
import subprocess
import sys
import sysconfig

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(PKG_DIR, "libsmla_b200.so")
NATIVE_SRC = os.path.join(PKG_DIR, "csrc", "native.cpp")
NATIVE_PATH = os.path.join(PKG_DIR, "_smla_native.so")
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-shared", "-Xcompiler", "-fPIC",
]


def sources():
    return sorted(glob.glob(os.path.join(PKG_DIR, "csrc", "*.cu")))


def _older(path: str, deps) -> bool:
    return not os.path.exists(path) or any(os.path.getmtime(d) > os.path.getmtime(path) for d in deps)


def _headers():
    return glob.glob(os.path.join(PKG_DIR, "..", "include", "*.h"))


def _run(cmd, verbose: bool) -> None:
    res = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"{cmd[0]} failed:\n" + res.stdout)
    if verbose:
        print(res.stdout)


def _stamp_path() -> str:
    return os.path.splitext(NATIVE_PATH)[0] + ".stamp"


def _stamped(cmd) -> bool:
    try:
        with open(_stamp_path()) as f:
            return f.read() == _stamp(cmd)
    except OSError:
        return False


def _stamp(cmd) -> str:
    import torch
    # (the tree may be moved)
    return "\n".join([f"torch {torch.__version__}", f"python {sys.version}"] + [os.path.relpath(c, PKG_DIR) if c in (NATIVE_PATH, NATIVE_SRC) else c for c in cmd])


def build_native(force: bool = False, verbose: bool = False) -> str:
    """Compile csrc/native.cpp; returns the extension's path.  Compiled again too when the torch or the Python that it was
    compiled against is another one, or the command: its layout of tensors is that torch's (the .stamp beside it says
    which)."""
    import torch
    from torch.utils import cpp_extension
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    libs = os.path.join(os.path.dirname(torch.__file__), "lib")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *(f"-I{p}" for p in cpp_extension.include_paths()), f"-I{sysconfig.get_paths()['include']}", f"-I{cuda}/include",
           "-o", NATIVE_PATH, NATIVE_SRC, f"-L{libs}", "-ltorch_python", "-ltorch_cpu", "-lc10_cuda", "-lc10", f"-L{cuda}/lib64", "-lcudart", "-ldl"]
    if not force and not _older(NATIVE_PATH, [NATIVE_SRC] + _headers()) and _stamped(cmd):
        return NATIVE_PATH
    _run(cmd, verbose)
    with open(_stamp_path(), "w") as f:
        f.write(_stamp(cmd))
    return NATIVE_PATH


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu under csrc/ into one shared library, and the extension; returns the library's path."""
    deps = sources() + glob.glob(os.path.join(PKG_DIR, "csrc", "*.cuh")) + _headers()
    if force or _older(LIB_PATH, deps):
        nvcc = os.environ.get("NVCC", "nvcc")
        _run([nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-o", LIB_PATH] + sources(), verbose)
    build_native(force, verbose)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
