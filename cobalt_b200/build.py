"""Build libcobalt_b200.so in-tree with nvcc for sm_100a.

    python -m cobalt_b200.build            # build if sources are newer than the library
    python -m cobalt_b200.build --force -v # rebuild and print ptxas resource usage
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libcobalt_b200.so")
SOURCES = ["cobalt_abi.cu", "compress_abi.cu"]
HEADERS = ["common.cuh", "decode_core.cuh", "walk_kernels.cuh", "gemv_kernel.cuh", "gemm_kernel.cuh", "glue_kernels.cuh", "staged_input.cuh", "compress_kernels.cuh",
           "prompt_attn.cuh",
           os.path.join("..", "..", "include", "cobalt_b200.h")]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; libcobalt_b200.so cannot be built")


def needs_build() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    files = [os.path.join(CSRC, f) for f in SOURCES + HEADERS]
    return any(os.path.getmtime(f) > t for f in files)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile the CUDA sources into the shared library and return its path."""
    if not force and not needs_build():
        return LIB
    cmd = [_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
           "--expt-relaxed-constexpr", "--threads", "0", "-shared", "-Xcompiler", "-fPIC",
           "-o", LIB] + [os.path.join(CSRC, s) for s in SOURCES]
    if verbose:
        cmd.insert(1, "-Xptxas")
        cmd.insert(2, "-v")
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose:
        sys.stderr.write(res.stderr)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + res.stdout + res.stderr)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
