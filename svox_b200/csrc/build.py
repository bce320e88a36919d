"""Compile the native library in-tree for sm_100a with nvcc, and its host extension.

    python -m svox_b200.csrc.build [--force] [--verbose]

Produces ``svox_b200/csrc/libsvox_b200.so``.  Default nvcc floating-point
behaviour is kept on purpose (no --use_fast_math, IEEE division and square
root): the kernels must reproduce the reference's arithmetic.
"""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "svox_b200.cu")
LIB = os.path.join(HERE, "libsvox_b200.so")
DEPS = ["svox_b200.cu", "common.cuh", "arith.cuh", "host.cuh", "binned.cuh", "tiles.cuh", "query.cuh", "render.cuh", "render_index.cuh",
        "render_queue.cuh", "render_back.cuh", "render_replay.cuh", "noalloc.cuh", "collective.cuh", "open_groups.h",
        os.path.join("..", "..", "include", "svox_b200.h")]


# the host side of the hot calls, a Python extension (host.cpp)
HOST_SRC = os.path.join(HERE, "host.cpp")
HOST_LIB = os.path.join(HERE, "_host.so")
HOST_DEPS = ["host.cpp", os.path.join("..", "..", "include", "svox_b200.h")]


def _stale(lib, deps):
    if not os.path.exists(lib):
        return True
    t = os.path.getmtime(lib)
    return any(os.path.getmtime(os.path.join(HERE, d)) > t for d in deps)


def _build_host():
    import sysconfig

    import torch
    from torch.utils import cpp_extension
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared",
           "-DTORCH_EXTENSION_NAME=_host", "-DTORCH_API_INCLUDE_EXTENSION_H",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    for d in [*cpp_extension.include_paths(), os.path.join(cuda, "include"),
              sysconfig.get_paths()["include"]]:
        cmd += ["-isystem", d]
    cmd += ["-o", HOST_LIB, HOST_SRC]
    for d in [*cpp_extension.library_paths(), os.path.join(cuda, "lib64")]:
        cmd += ["-L" + d]
    cmd += ["-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python",
            "-lcudart"]
    subprocess.run(cmd, check=True)


def build(force=False, verbose=False):
    if force or _stale(HOST_LIB, HOST_DEPS):
        _build_host()
    if not force and not _stale(LIB, DEPS):
        return LIB
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    cmd = [nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3",
           "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-o", LIB, SRC]
    if verbose:
        cmd.insert(1, "-Xptxas")
        cmd.insert(2, "-v")
    subprocess.run(cmd, check=True)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
