"""Ahead-of-time build of the native library for sm_100a.

    python qfactory-ae_b200/build.py [--force] [--verbose]

Compiles every csrc/*.cu with nvcc (one process per file, in parallel) and links
lib/libqfactory_b200.so.  The library only depends on the statically linked CUDA
runtime, so it loads on a machine without a GPU (calls then fail with a CUDA error).
csrc/qfb_torch.cpp, the CPython module that calls the library on torch tensors, is
compiled with g++ against the installed torch's headers into lib/_qfb_torch.so; without
torch only the library is built, which is all that the C ABI needs.
A source newer than its library triggers a rebuild, and another torch or Python one of the module.
"""
from __future__ import annotations

import glob
import importlib.metadata
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB_DIR = os.path.join(HERE, "lib")
LIB = os.path.join(LIB_DIR, "libqfactory_b200.so")
TORCH_SRC = os.path.join(CSRC, "qfb_torch.cpp")
TORCH_LIB = os.path.join(LIB_DIR, "_qfb_torch.so")
TORCH_FOR = os.path.join(OBJ, "_qfb_torch.for")   # the torch and the Python it was built against
HEADER = os.path.join(os.path.dirname(HERE), "include", "qfactory_b200.h")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "--expt-relaxed-constexpr", "--extended-lambda",
    "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    raise RuntimeError("nvcc not found")


def sources() -> list[str]:
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _deps() -> list[str]:
    return sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.h")) + [HEADER]


def is_stale() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    return any(os.path.getmtime(d) > t for d in _deps())


def _torch_version() -> str | None:
    try:   # (without importing it, which takes seconds)
        return importlib.metadata.version("torch")
    except importlib.metadata.PackageNotFoundError:
        return None


def torch_module_is_stale(version: str) -> bool:
    """Older than its sources, or built for another torch or Python than the ones here."""
    if not os.path.exists(TORCH_LIB) or any(os.path.getmtime(d) > os.path.getmtime(TORCH_LIB) for d in (TORCH_SRC, HEADER)):
        return True
    try:
        with open(TORCH_FOR) as f:
            return f.read() != _built_for(version)
    except OSError:
        return True


def _built_for(version: str) -> str:
    return f"torch {version}, {sysconfig.get_config_var('SOABI')}"


def build_torch_module(force: bool = False, verbose: bool = False) -> str | None:
    version = _torch_version()
    if version is None:
        sys.stderr.write("torch is not installed: the library is built, the module for torch tensors is not\n")
        return None
    if not force and not torch_module_is_stale(version):
        return TORCH_LIB
    import torch

    os.makedirs(LIB_DIR, exist_ok=True)
    os.makedirs(OBJ, exist_ok=True)
    root = os.path.dirname(torch.__file__)
    cuda_inc = os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include")
    tmp = TORCH_LIB + ".tmp"
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           "-I" + os.path.join(root, "include"), "-I" + os.path.join(root, "include", "torch", "csrc", "api", "include"),
           "-I" + sysconfig.get_paths()["include"], "-I" + (cuda_inc if os.path.isdir(cuda_inc) else "/usr/local/cuda/include"),
           TORCH_SRC, "-o", tmp, "-L" + os.path.join(root, "lib"), "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed on {TORCH_SRC}")
    os.replace(tmp, TORCH_LIB)
    with open(TORCH_FOR, "w") as f:
        f.write(_built_for(version))
    return TORCH_LIB


def build(force: bool = False, verbose: bool = False) -> str:
    lib = build_library(force, verbose)
    build_torch_module(force, verbose)
    return lib


def build_library(force: bool = False, verbose: bool = False) -> str:
    if not force and not is_stale():
        return LIB
    os.makedirs(OBJ, exist_ok=True)
    os.makedirs(LIB_DIR, exist_ok=True)
    nvcc = _nvcc()
    extra = ["-Xptxas", "-v"] if verbose else []
    extra += os.environ.get("QFB_NVCC_EXTRA", "").split()

    def compile_one(src: str) -> str:
        obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
        cmd = [nvcc, *NVCC_FLAGS, *extra, "-c", src, "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if verbose or r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}")
        return obj

    with ThreadPoolExecutor(max_workers=min(8, len(sources()))) as ex:
        objs = list(ex.map(compile_one, sources()))
    tmp = LIB + ".tmp"
    cmd = [nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-o", tmp, *objs]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError("link failed")
    os.replace(tmp, LIB)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
