"""Builds the CUDA library (C ABI in include/ragged_dot_b200.h) in-tree with nvcc for sm_100a.

    python -m gpu_ragged_dot_b200.build [--force]

The shared object lands next to this file as ``librd_b200.so``; nvcc cross-compiles, so no
GPU is needed to build.  ``_rd_host.so`` beside it is the native host path of the torch layer
(csrc/rd_torch.cpp), linked against it and against torch.
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC_DIR = os.path.join(PKG_DIR, "csrc")
LIB_PATH = os.path.join(PKG_DIR, "librd_b200.so")
HOST_PATH = os.path.join(PKG_DIR, "_rd_host.so")
HOST_SOURCE = os.path.join(CSRC_DIR, "rd_torch.cpp")
HEADER = os.path.join(PKG_DIR, "..", "include", "ragged_dot_b200.h")
SOURCES = ["rd_api.cu"]

NVCC_FLAGS = [
    "-gencode",
    "arch=compute_100a,code=sm_100a",
    "-lineinfo",
    "-O3",
    "-std=c++17",
    "--shared",
    "-Xcompiler",
    "-fPIC",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found: cannot build librd_b200.so")
    return exe


def _stale() -> bool:
    if not os.path.exists(LIB_PATH):
        return True
    built = os.path.getmtime(LIB_PATH)
    deps = [os.path.join(CSRC_DIR, f) for f in os.listdir(CSRC_DIR) if f.endswith((".cu", ".cuh", ".h"))]
    deps.append(os.path.join(PKG_DIR, "..", "include", "ragged_dot_b200.h"))
    return any(os.path.getmtime(d) > built for d in deps if os.path.exists(d))


def build_library(force: bool = False, verbose: bool = False) -> str:
    """Compile librd_b200.so if it is missing or older than its sources; return its path."""
    if not force and not _stale():
        return LIB_PATH
    cmd = [_nvcc(), *NVCC_FLAGS]
    if verbose:
        cmd += ["-Xptxas", "-v"]
    cmd += ["-o", LIB_PATH] + [os.path.join(CSRC_DIR, s) for s in SOURCES]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError(f"nvcc failed ({proc.returncode}):\n{proc.stdout}\n{proc.stderr}")
    if verbose:
        sys.stderr.write(proc.stderr)
    return LIB_PATH


def build_host(force: bool = False) -> str:
    """Compile _rd_host.so if it is missing or older than its sources or the installed torch; return its path."""
    import sysconfig

    import torch
    from torch.utils import cpp_extension

    deps = [HOST_SOURCE, HEADER, torch.version.__file__]  # built for one torch's headers and libraries
    if not force and os.path.exists(HOST_PATH) and all(os.path.getmtime(d) <= os.path.getmtime(HOST_PATH) for d in deps):
        return HOST_PATH

    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    cmd = [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden",
           "-DTORCH_EXTENSION_NAME=_rd_host", "-DTORCH_API_INCLUDE_EXTENSION_H",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    for path in [*cpp_extension.include_paths(), os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]:
        cmd += ["-isystem", path]
    cmd += ["-o", HOST_PATH, HOST_SOURCE, f"-L{PKG_DIR}", "-lrd_b200", "-Wl,-rpath,$ORIGIN"]
    for path in cpp_extension.library_paths():
        cmd += [f"-L{path}", f"-Wl,-rpath,{path}"]
    cmd += ["-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_python"]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError(f"g++ failed ({proc.returncode}):\n{proc.stdout}\n{proc.stderr}")
    return HOST_PATH


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
    print(build_host(force="--force" in sys.argv))
