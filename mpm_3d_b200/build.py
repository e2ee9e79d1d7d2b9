"""Builds the CUDA library libmpm_b200.so in-tree (sm_100a only).

``python -m mpm_3d_b200.build`` or ``build()`` from Python. The library is
written to ``mpm_3d_b200/lib/`` so that it travels with the source tree.
"""
from __future__ import annotations

import os
import subprocess
import sys
import tempfile
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
LIB_DIR = os.path.join(HERE, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libmpm_b200.so")
HEADERS_DIR = os.path.join(HERE, "csrc")

# One object file each (source, defines, further flags): the engine with its
# small kernels, and the fused kernel's instantiations in groups, which compile
# in parallel (90 s on 8 cores). nvcc's -split-compile is not used: what it makes
# of a kernel differs from one run to the next (the column's step took 382 or 408
# us with libraries built from the same source by the same command).
UNITS = [("fused_kernels.cu", {"MPM_STAGED_DET": "0", "MPM_POINT": pt}, []) for pt in ("float", "double")]
UNITS += [("fused_kernels.cu", {"MPM_LEAN_CAP": str(cap), "MPM_POINT": pt}, [])
          for pt in ("double", "float") for cap in (512, 256, 128)]
# the deterministic kernel with fewer spills (49,152-point column 72.3 -> 62.7 us
# per step); the other kernels are as fast without, or faster (two-body collision
# 108 us, 113 with it)
UNITS += [("fused_kernels.cu", {"MPM_STAGED_DET": "1", "MPM_POINT": "double"},
           ["-Xptxas", "--register-usage-level=0"]),
          ("api.cu", {}, [])]

NVCC_FLAGS = [
    "-ccbin", "/usr/bin/g++",
    "-std=c++17",
    "-O3",
    "-lineinfo",
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-Xcompiler", "-fPIC",
    "-Xfatbin", "-compress-all",
]


def _newest_source_mtime() -> float:
    paths = [os.path.abspath(__file__), os.path.join(ROOT, "include", "mpm_b200.h")]
    for name in os.listdir(HEADERS_DIR):
        paths.append(os.path.join(HEADERS_DIR, name))
    return max(os.path.getmtime(p) for p in paths)


def nvcc() -> str:
    cand = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    return cand if os.path.exists(cand) else "nvcc"


def build(force: bool = False, verbose: bool = False) -> str:
    """Compiles the library if it is missing or older than its sources."""
    if not force and os.path.exists(LIB_PATH) and os.path.getmtime(LIB_PATH) >= _newest_source_mtime():
        return LIB_PATH
    os.makedirs(LIB_DIR, exist_ok=True)
    flags = NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else [])
    tmp = LIB_PATH + ".tmp"
    with tempfile.TemporaryDirectory() as objects:

        def compile_unit(i: int) -> str:
            source, defines, more = UNITS[i]
            obj = os.path.join(objects, f"{i}.o")
            subprocess.check_call([nvcc()] + flags + more + [f"-D{k}={v}" for k, v in defines.items()] +
                                  ["-c", os.path.join(HEADERS_DIR, source), "-o", obj])
            return obj

        with ThreadPoolExecutor(os.cpu_count() or 1) as pool:
            objs = list(pool.map(compile_unit, range(len(UNITS))))
        subprocess.check_call([nvcc()] + NVCC_FLAGS + ["-shared"] + objs + ["-o", tmp])
    os.replace(tmp, LIB_PATH)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
