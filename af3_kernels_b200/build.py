"""Builds ``libaf3k.so`` (nvcc, sm_100a) and ``_host.so`` (g++, torch headers) in-tree.

Usage: ``python -m af3_kernels_b200.build [--force]``.  nvcc cross-compiles, so this works on a
host without a GPU; the resulting library needs a compute-capability-10.x device to run.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

_HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(_HERE, "csrc")
LIB_PATH = os.path.join(_HERE, "libaf3k.so")
SOURCES = [os.path.join(CSRC, "af3k_capi.cu")]
HEADERS = [
    os.path.join(CSRC, "attn_sm100.cuh"),
    os.path.join(CSRC, "pair_bias_sm100.cuh"),
    os.path.join(CSRC, "grid_sm100.cuh"),
    os.path.join(CSRC, "ptx_sm100.cuh"),
    os.path.join(CSRC, "token_sm100.cuh"),
    os.path.join(_HERE, "..", "include", "af3k.h"),
]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-shared", "-Xcompiler", "-fPIC",
    "-cudart", "shared",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; libaf3k.so cannot be built")
    return exe


# the host path on at::Tensor: an extension module beside the binding (it looks the library's entry
# points up at run time, so it does not link against libaf3k.so)
HOST_SRC = os.path.join(CSRC, "host_torch.cpp")
HOST_PATH = os.path.join(_HERE, "_host.so")


def _older(path, sources) -> bool:
    if not os.path.exists(path):
        return True
    t = os.path.getmtime(path)
    return any(os.path.getmtime(f) > t for f in sources)


def is_stale() -> bool:
    return _older(LIB_PATH, SOURCES + HEADERS) or _older(HOST_PATH, [HOST_SRC, HEADERS[-1]])


def _run(cmd, what, verbose):
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
    if res.returncode != 0:
        raise RuntimeError(f"building {what} failed")


def build_host(verbose: bool = False) -> None:
    import sysconfig

    import torch

    tdir = os.path.dirname(torch.__file__)
    inc = [os.path.join(tdir, "include"), os.path.join(tdir, "include", "torch", "csrc", "api", "include"),
           os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include"), sysconfig.get_paths()["include"]]
    lib = os.path.join(tdir, "lib")
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_host",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}"]
    cmd += [f"-I{d}" for d in inc] + [HOST_SRC, "-o", HOST_PATH, f"-L{lib}"]
    cmd += ["-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python", "-ldl"]
    _run(cmd, "_host.so", verbose)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compiles what is missing or older than its sources; returns the library's path."""
    if force or _older(LIB_PATH, SOURCES + HEADERS):
        _run([_nvcc()] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-o", LIB_PATH] + SOURCES, "libaf3k.so", verbose)
    if force or _older(HOST_PATH, [HOST_SRC, HEADERS[-1]]):
        build_host(verbose)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
