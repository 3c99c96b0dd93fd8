"""Builds libcame_b200.so in-tree with nvcc for sm_100a, and the host module _host.so (g++, against torch's headers) that
links to it.  No JIT cache.

    python came_b200/_build.py [--force] [--verbose]
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
INCLUDE = os.path.join(ROOT, "include")
OBJDIR = os.path.join(CSRC, "build")
LIB = os.path.join(PKG, "libcame_b200.so")
HOST = os.path.join(PKG, "_host.so")
SOURCES = ["capi.cu", "codec.cu", "factored.cu", "fast_tile8.cu", "fp_wide.cu", "fused_ma.cu", "fused_sq.cu", "generic.cu", "nd.cu", "nd_fixed.cu", "noalloc.cu"]
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
NVCC_FLAGS = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC", "-I", INCLUDE, "-I", CSRC]
NVCC_FLAGS += os.environ.get("CAME_B200_NVCC_FLAGS", "").split()   # build-time experiment switches, e.g. -DCAME_TUNE


def find_nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC or put it on PATH")


def _newest_source_mtime() -> float:
    paths = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h", ".cpp"))]
    paths.append(os.path.join(INCLUDE, "came_b200.h"))
    return max(os.path.getmtime(p) for p in paths)


def is_stale() -> bool:
    built = [os.path.getmtime(p) for p in (LIB, HOST) if os.path.exists(p)]
    return len(built) < 2 or min(built) < _newest_source_mtime()


def build_host() -> None:
    """The CPython extension module: plain g++ with the include and library paths of the installed torch."""
    import torch
    from torch.utils import cpp_extension
    cuda = os.path.dirname(os.path.dirname(find_nvcc()))
    libs = os.path.join(os.path.dirname(torch.__file__), "lib")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", "-w",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", "-I", INCLUDE,
           "-I", sysconfig.get_path("include"), "-I", os.path.join(cuda, "include")]
    for inc in cpp_extension.include_paths():
        cmd += ["-isystem", inc]
    tmp = HOST + ".tmp"
    cmd += [os.path.join(CSRC, "host.cpp"), "-o", tmp, "-L", PKG, "-l:libcame_b200.so", "-Wl,-rpath,$ORIGIN", "-L", libs,
            "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"g++ failed on host.cpp:\n{res.stdout}\n{res.stderr}")
    os.replace(tmp, HOST)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compiles every translation unit for sm_100a, links the shared library and the host module; returns the library's path."""
    if not force and not is_stale():
        return LIB
    nvcc = find_nvcc()
    os.makedirs(OBJDIR, exist_ok=True)
    extra = ["-Xptxas", "-v"] if verbose else []

    def compile_one(src: str) -> str:
        obj = os.path.join(OBJDIR, src.replace(".cu", ".o"))
        cmd = [nvcc, *ARCH, *NVCC_FLAGS, *extra, "-c", os.path.join(CSRC, src), "-o", obj]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{res.stdout}\n{res.stderr}")
        if verbose:
            sys.stderr.write(res.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=len(SOURCES)) as ex:
        objs = list(ex.map(compile_one, SOURCES))
    tmp = LIB + ".tmp"
    res = subprocess.run([nvcc, *ARCH, "-shared", "-o", tmp, *objs], capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    os.replace(tmp, LIB)
    build_host()
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
