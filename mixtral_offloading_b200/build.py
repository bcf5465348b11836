"""Builds the C-ABI library (hand-written sm_100a CUDA + the C++ cache runtime) and the Python extension over it in-tree.

    python -m mixtral_offloading_b200.build [--force]

One compiler invocation per source, in parallel, no build system.  The outputs, libhqq_moe_b200.so and _host.so, sit
beside this file.
"""
from __future__ import annotations

import glob
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libhqq_moe_b200.so")
HOST_SRC = os.path.join(HERE, "native", "host.cpp")
HOST = os.path.join(HERE, "_host.so")

NVCC_FLAGS = [
    "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-Xcompiler", "-fPIC",
]
OBJ = os.path.join(HERE, "..", "build", "obj")


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cpp")))


def _headers():
    return glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.h")) + glob.glob(os.path.join(HERE, "..", "include", "*.h"))


def _stale(target, deps):
    return not os.path.exists(target) or any(os.path.getmtime(p) > os.path.getmtime(target) for p in deps)


def _run(cmd, verbose=False):
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("compilation failed:\n" + " ".join(cmd) + "\n" + res.stdout + res.stderr)
    if verbose:
        print(res.stderr)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compiles what is out of date (one object per source, in parallel) and links the library."""
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    os.makedirs(OBJ, exist_ok=True)
    jobs = []
    for src in sources():
        obj = os.path.join(OBJ, os.path.basename(src) + ".o")
        if force or _stale(obj, [src] + _headers()):
            jobs.append([nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", "-o", obj, src])
    with ThreadPoolExecutor(os.cpu_count() or 1) as pool:
        list(pool.map(lambda cmd: _run(cmd, verbose), jobs))
    objs = [os.path.join(OBJ, os.path.basename(src) + ".o") for src in sources()]
    if jobs or _stale(LIB, objs):
        _run([nvcc] + NVCC_FLAGS + ["-shared", "-o", LIB] + objs)
    if jobs or force or _stale(HOST, [HOST_SRC, LIB] + _headers()):
        _build_host(verbose)
    return LIB


def _build_host(verbose):
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.join(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")), "..")
    _run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
          f"-I{root}/include", f"-I{root}/include/torch/csrc/api/include", f"-I{sysconfig.get_paths()['include']}",
          f"-I{cuda}/include", "-o", HOST, HOST_SRC, f"-L{HERE}", "-l:" + os.path.basename(LIB), f"-L{root}/lib", "-lc10",
          "-ltorch_cpu", "-ltorch_python", "-lc10_cuda", "-Wl,-rpath,$ORIGIN"], verbose)


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
