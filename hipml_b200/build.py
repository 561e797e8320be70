"""Builds libhipml_cuda.so (the C-ABI library) in-tree with nvcc for sm_100a."""
from __future__ import annotations

import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "lib")
LIB = os.path.join(LIB_DIR, "libhipml_cuda.so")
CALLS = os.path.join(LIB_DIR, "_hipml_calls.so")   # CPython view of the launchers

SOURCES = [
    "device_api.cu",
    "kv_encode.cu",
    "attn_decode.cu",
    "attn_decode_tc.cu",
    "attn_decode_warps.cu",
    "attn_decode_cols.cu",
    "attn_decode_f32.cu",
    "decode_static.cu",
    "decode_exchange.cu",
    "attn_front.cu",
    "attn_chunk_scalar.cu",
    "attn_chunk_small.cu",
    "attn_chunk_tc.cu",
    "launchers.cu",
]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
]


def nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.sep not in cand or os.path.exists(cand)):
            return cand
    raise RuntimeError("nvcc not found")


def _stale() -> bool:
    if not os.path.exists(LIB) or not os.path.exists(CALLS):
        return True
    t = min(os.path.getmtime(LIB), os.path.getmtime(CALLS))
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)]
    deps.append(os.path.join(os.path.dirname(HERE), "include", "hipml_cuda.h"))
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu into one shared library and the Python call module; returns the library's path."""
    if not force and not _stale():
        return LIB
    os.makedirs(LIB_DIR, exist_ok=True)
    objs = []
    for src in SOURCES:
        obj = os.path.join(LIB_DIR, src.replace(".cu", ".o"))
        cmd = [nvcc(), *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        subprocess.check_call(cmd)
        objs.append(obj)
    subprocess.check_call([nvcc(), "-shared", "-o", LIB, *objs, "-gencode",
                           "arch=compute_100a,code=sm_100a"])
    # (links to the library beside it: the process holds one copy, whoever loads it first)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-Wall",
                           "-I", sysconfig.get_paths()["include"], os.path.join(CSRC, "py_calls.cpp"),
                           "-o", CALLS, "-L", LIB_DIR, "-l:libhipml_cuda.so", "-Wl,-rpath,$ORIGIN"])
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
