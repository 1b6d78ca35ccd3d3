"""Builds in-tree: libfrnn_b200.so (the C-ABI launch library, nvcc for sm_100a) and _frnn_host.so (the native host
path of a call, g++ against PyTorch's headers)."""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
LIB = os.path.join(HERE, "libfrnn_b200.so")
SRC = os.path.join(HERE, "csrc", "frnn_shim.cu")
DEPS = [SRC, os.path.join(HERE, "..", "include", "frnn.h")]
HOST_LIB = os.path.join(HERE, "_frnn_host.so")
HOST_SRC = os.path.join(HERE, "csrc", "frnn_host.cpp")


def nvcc_path() -> str:
    for cand in (os.environ.get("CUDA_HOME", "") + "/bin/nvcc", "/usr/local/cuda/bin/nvcc", shutil.which("nvcc") or ""):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; cannot build libfrnn_b200.so")


def up_to_date(lib: str = LIB, deps=DEPS) -> bool:
    if not os.path.exists(lib):
        return False
    t = os.path.getmtime(lib)
    return all(os.path.getmtime(d) <= t for d in deps if os.path.exists(d))


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and up_to_date():
        return LIB
    cmd = [nvcc_path(), "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
           "-shared", "-Xcompiler", "-fPIC", "-Xptxas", "-v", "-cudart", "static",
           "-o", LIB, SRC, "-ldl"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or r.returncode:
        sys.stderr.write(r.stdout + r.stderr)
    if r.returncode:
        raise RuntimeError("building libfrnn_b200.so failed:\n" + r.stderr)
    return LIB


def build_host(force: bool = False) -> str:
    """The native host path.  Needs PyTorch's headers and the CUDA toolkit's, no GPU."""
    if not force and up_to_date(HOST_LIB, [HOST_SRC]):
        return HOST_LIB
    import sysconfig
    import torch
    from torch.utils.cpp_extension import include_paths, library_paths
    cuda = os.path.dirname(os.path.dirname(nvcc_path()))
    incs = include_paths() + [os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    tmp = f"{HOST_LIB}.{os.getpid()}.tmp"
    cmd = [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden",
           "-DTORCH_EXTENSION_NAME=_frnn_host", "-DTORCH_API_INCLUDE_EXTENSION_H",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *[f"-isystem{i}" for i in incs], HOST_SRC, "-o", tmp,
           *[f"-L{p}" for p in library_paths()], "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode:
        raise RuntimeError("building _frnn_host.so failed:\n" + r.stderr[-6000:])
    os.replace(tmp, HOST_LIB)
    return HOST_LIB


if __name__ == "__main__":
    print(build_host(force="--force" in sys.argv))
    print(build(force="--force" in sys.argv, verbose=True))
