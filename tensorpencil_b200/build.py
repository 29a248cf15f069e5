"""Builds ``libtpb200.so`` in-tree with nvcc for sm_100a.

    python -m tensorpencil_b200.build [--force] [--verbose]

The library is plain CUDA C++ behind a C ABI (``include/tpb200.h``); it links the
static CUDA runtime and resolves the one driver entry point it needs at run
time, so it loads on a machine without a GPU or driver.
"""
from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys
import sysconfig

from ._lib import CALL_PATH

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
OUT_DIR = os.path.join(PKG, "lib")
LIB = os.path.join(OUT_DIR, "libtpb200.so")
OBJ_DIR = os.path.join(OUT_DIR, "obj")
PYCALL_SRC = os.path.join(CSRC, "pycall.c")

SOURCES = ["api.cu", "prep.cu", "prep_fused.cu", "gemm_i8.cu", "gemm2_i8.cu", "gemm_splitk.cu", "gemm_w4.cu", "qgemv.cu", "qgemv_mma.cu", "qgemv_k.cu", "qgemv_kmma.cu", "offload.cu", "peer.cu", "attn.cu"]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC,-O3,-Wall,-Wno-unused-function",
    "--expt-relaxed-constexpr",
    "-I", os.path.join(ROOT, "include"), "-I", CSRC,
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; libtpb200.so cannot be built")
    return exe


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build_pycall(out: str, lib_dir: str) -> bool:
    """The CPython entry to the hot calls (csrc/pycall.c) for the running interpreter, linked to lib_dir/libtpb200.so, by the compiler that
    nvcc drives.  Without Python's headers it is left out, and the calls go through ctypes (_lib.load_calls)."""
    inc = sysconfig.get_paths()["include"]
    if not os.path.exists(os.path.join(inc, "Python.h")):
        sys.stderr.write(f"{inc}/Python.h not found: {os.path.basename(out)} is not built, calls go through ctypes\n")
        return False
    subprocess.run([_nvcc(), "-O2", "-Xcompiler", "-fPIC,-Wall", "-shared", "-cudart", "none", "-I", inc,
                    "-I", os.path.join(ROOT, "include"), PYCALL_SRC, "-o", out, "-L", lib_dir, "-Xlinker", "-l:libtpb200.so",
                    "-Xlinker", "-rpath,$ORIGIN"], check=True)
    return True


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ_DIR, exist_ok=True)
    headers = [os.path.join(ROOT, "include", "tpb200.h")] + [
        os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".h", ".cuh"))]
    nvcc = _nvcc()
    # nvcc must drive a host compiler it supports; the image's default gcc works.
    env = dict(os.environ)
    objs = []
    procs = []
    for src in SOURCES:
        s = os.path.join(CSRC, src)
        o = os.path.join(OBJ_DIR, src.replace(".cu", ".o"))
        objs.append(o)
        if force or _stale(o, [s] + headers):
            cmd = [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", s, "-o", o]
            procs.append((src, subprocess.Popen(cmd, env=env, stdout=subprocess.PIPE,
                                                stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0 or verbose:
            sys.stderr.write(f"--- nvcc {src} ---\n{out}\n")
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed")
    if force or procs or _stale(LIB, objs):
        cmd = [nvcc, "-shared", "-o", LIB] + objs + ["-cudart", "static",
                                                     "-Xlinker", "--no-undefined"]
        subprocess.run(cmd, check=True, env=env)
    if force or _stale(CALL_PATH, [PYCALL_SRC, headers[0]]):
        build_pycall(CALL_PATH, OUT_DIR)
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose))
