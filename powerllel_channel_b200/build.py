"""Build recipe of libpowerllel_b200.so (nvcc, sm_100a), in-tree.

    python -m powerllel_channel_b200.build
"""
from __future__ import annotations

import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libpowerllel_b200.so")
SOURCES = ["ppe.cu", "fft_len1.cu", "fft_len2.cu", "fft_len3.cu", "fft_len4.cu", "stencil.cu", "rk_fused.cu", "rk_mixed.cu", "channel.cu", "adjoint.cu", "monitor.cu"]
HEADERS = ["common.cuh", "fft.cuh", "fft_kernels.cuh", "fft_launch.cuh", "ppe.cuh", "stencil.cuh", "stencil_rhs.cuh", "tmem.cuh", "trid_tables.h", "channel.cuh"]

NVCC_FLAGS = [
    "-std=c++17", "-O3", "-lineinfo", "--threads", "0",
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-Xcompiler", "-fPIC", "-shared",
]


def _nvcc() -> str:
    for c in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if c and (os.path.sep not in c or os.path.exists(c)):
            return c
    return "nvcc"


def stale() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = [os.path.join(CSRC, f) for f in SOURCES + HEADERS] + [os.path.join(ROOT, "include", "powerllel_b200.h")]
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not stale():
        return LIB
    cmd = [_nvcc(), *NVCC_FLAGS, "-I", os.path.join(ROOT, "include"), "-o", LIB + ".tmp",
           *[os.path.join(CSRC, f) for f in SOURCES]]
    if verbose:
        print(" ".join(cmd), flush=True)
    subprocess.run(cmd, check=True)
    os.replace(LIB + ".tmp", LIB)
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose=True)
    print(LIB)
