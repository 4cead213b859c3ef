"""Ahead-of-time build of libb200moe.so (sm_100a only) with nvcc; no JIT cache, the library stays in-tree.

    python -m kernelschema_b200.build [--force] [--verbose]
"""
from __future__ import annotations

import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libb200moe.so")
SHIM = os.path.join(HERE, "_b200moe_shim.so")
SOURCES = ["quantize.cu", "router.cu", "route_map.cu", "gather.cu", "finalize.cu", "gemm_nvfp4.cu", "gemm_w4a16.cu", "gemm_w4a16_decode.cu", "gemm_w4a16_expand.cu", "ep_exchange.cu", "api.cu"]
HEADERS = ["kernels.cuh", "ptx.cuh", "quantize.cuh", "topk.cuh", "w4a16.cuh", os.path.join("..", "..", "include", "b200moe.h")]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC",
              "-Xptxas", "-v"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.sep not in cand or os.path.exists(cand)):
            return cand
    raise RuntimeError("nvcc not found")


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every CUDA source for sm_100a and link the shared library. Returns its path."""
    nvcc = _nvcc()
    objdir = os.path.join(HERE, "build")
    os.makedirs(objdir, exist_ok=True)
    headers = [os.path.join(CSRC, h) for h in HEADERS]

    def compile_one(src: str) -> str:
        obj = os.path.join(objdir, src.replace(".cu", ".o"))
        path = os.path.join(CSRC, src)
        if force or _stale(obj, [path] + headers):
            cmd = [nvcc, *NVCC_FLAGS, "-c", path, "-o", obj]
            res = subprocess.run(cmd, capture_output=True, text=True)
            with open(obj + ".log", "w") as f:
                f.write(" ".join(cmd) + "\n" + res.stdout + res.stderr)
            if res.returncode != 0:
                raise RuntimeError(f"nvcc failed on {src}:\n{res.stderr}")
            if verbose:
                print(res.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=min(8, len(SOURCES))) as ex:
        objs = list(ex.map(compile_one, SOURCES))
    if force or _stale(LIB, objs):
        cmd = [nvcc, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a"]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError("link failed:\n" + res.stderr)
    build_shim(force)
    return LIB


def build_shim(force: bool = False) -> str:
    """Compile the pybind11 shim (plain C++, links against the in-tree libb200moe.so through $ORIGIN)."""
    import sysconfig
    import pybind11
    src = os.path.join(CSRC, "shim.cpp")
    if force or _stale(SHIM, [src, LIB, os.path.join(CSRC, "..", "..", "include", "b200moe.h")]):
        cmd = ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden", "-I", pybind11.get_include(), "-I",
               sysconfig.get_paths()["include"], src, "-o", SHIM, "-L", HERE, "-lb200moe", "-Wl,-rpath,$ORIGIN"]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError("shim build failed:\n" + res.stderr)
    return SHIM


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
