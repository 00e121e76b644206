"""Build the CUDA library in-tree: mgpoisson2d_b200/libmgp2d.so (sm_100a).

    python -m mgpoisson2d_b200.build [--force]

-fmad=false keeps every FP64 product and sum separately rounded, so each cell
the kernels compute is bit-identical to the Fortran loop body it restates.
"""
from __future__ import annotations

import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
LIB = os.path.join(HERE, "libmgp2d.so")
SOURCES = ["mgp_kernels.cu", "mgp_sweep.cu", "mgp_ddsweep.cu", "mgp_bottom.cu", "mgp_host.cu", "mgp_noalloc.cu", "mgp_batch.cu", "mgp_geometry.cu",
           "mgp_lockstep.cu"]
HEADERS = ["mgp_core.cuh", "mgp_kernels.cuh", "mgp_stage.cuh", "mgp_sweep.cuh", "mgp_ddsweep.cuh"]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-lineinfo", "-std=c++17", "-fmad=false",
    "-Xcompiler", "-fPIC,-O3", "-shared",
]


def _nvcc() -> str:
    for c in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if c and (os.path.sep not in c or os.path.exists(c)):
            return c
    return "nvcc"


def stale() -> bool:
    if not os.path.exists(LIB):
        return True
    deps = [os.path.join(CSRC, f) for f in SOURCES + HEADERS] + [os.path.join(INCLUDE, "mgp2d.h")]
    t = os.path.getmtime(LIB)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not stale():
        return LIB
    cmd = [_nvcc(), *NVCC_FLAGS, "-I", INCLUDE, "-o", LIB] + [os.path.join(CSRC, s) for s in SOURCES]
    if verbose:
        print(" ".join(cmd))
    subprocess.run(cmd, check=True)
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose=True)
