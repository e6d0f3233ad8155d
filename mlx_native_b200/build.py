"""Builds the CUDA library in-tree: mlx_native_b200/libmlxn_b200.so (sm_100a only).

Run as `python -m mlx_native_b200.build` or through `__graft_entry__.build()`.  nvcc
cross-compiles for sm_100a without a GPU; the built library is loaded with ctypes.
"""
from __future__ import annotations

import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libmlxn_b200.so")
SOURCES = ["runtime.cu", "qmv.cu", "qmv_tc.cu", "qmv_mma.cu", "qmv_split.cu", "qmv_split_q4_0.cu", "qmv_split_q8_0.cu",
           "qmv_split_q4_k.cu", "qmv_split_q5_k.cu", "qmv_split_q6_k.cu", "qmv_wide.cu", "qmm.cu", "qmm_duo.cu", "moe.cu"]
HEADERS = ["common.cuh", "dequant.cuh", "qmm.cuh", "mma_f16.cuh", "ptx.cuh", "qmv_split.cuh", "tensor_map.cuh", os.path.join("..", "..", "include", "mlxn_b200.h")]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17",
    "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def needs_build() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = [os.path.join(CSRC, s) for s in SOURCES + HEADERS]
    return any(os.path.exists(d) and os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not needs_build():
        return LIB
    flags = list(NVCC_FLAGS) + os.environ.get("MLXN_NVCC_EXTRA", "").split()   # e.g. -DMLXN_TC_TRACE for experiments
    objs = []
    procs = []
    for s in SOURCES:
        obj = os.path.join(CSRC, s.replace(".cu", ".o"))
        objs.append(obj)
        cmd = [_nvcc(), *flags, "-c", os.path.join(CSRC, s), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas")
            cmd.insert(2, "-v")
        procs.append((s, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for s, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0:
            failed = True
            sys.stderr.write(f"nvcc failed on {s}:\n{out}\n")
        elif verbose:
            sys.stderr.write(out)
    if failed:
        raise RuntimeError("nvcc failed; see messages above")
    subprocess.check_call([_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-o", LIB, *objs])
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
