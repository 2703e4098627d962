"""Builds libukgpu.so (the C-ABI library with the CUDA smoothers) in-tree.

nvcc compiles every translation unit for sm_103a only, in parallel, and links
them into ultimate_kalman_gb300/libukgpu.so.  Run directly or through
``__graft_entry__.build()``.
"""
from __future__ import annotations

import concurrent.futures as cf
import glob
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
BUILD = os.path.join(HERE, "_build")
LIB = os.path.join(HERE, "libukgpu.so")

ARCH = ["-gencode", "arch=compute_103a,code=sm_103a"]
SOURCES = ["oddeven.cu", "associative.cu", "builder.cu", "filter.cu", "profiling.cu", "host_api.cpp", "matrix_ops.c"]
# oddeven.cu's kernels by arithmetic type, a compilation each
PARTS = {"oddeven.cu": [("f32", "float"), ("f64", "double"), ("df", "ukg_df::dd")]}
# --split-compile=0: nvcc optimizes a translation unit's kernels in parallel on every
# core.  That gives other code at every build of the same source (the residual of 6
# states took 46 or 63 us, the scans of 48 states 50 or 60 ms), so what it does not speed
# up every time is compiled without: the FP32 and double-float parts (pairs of 128
# states 8.8 ms with, 8.1 without) and the associative smoother.  The FP64 part keeps it:
# its back-substitutions of 16 states and of 65 and more are 20 % slower without.
SPLIT = ["--split-compile=0"]
WHOLE = ("associative.cu",)


def nvcc():
    for c in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if c and os.path.exists(c):
            return c
    raise FileNotFoundError("nvcc not found")


def _compile(unit, verbose):
    src, name, flags = unit
    out = os.path.join(BUILD, name + ".o")
    inc = ["-I", os.path.join(REPO, "include"), "-I", CSRC]
    if src.endswith(".cu"):
        cmd = [nvcc(), *ARCH, "-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC", *inc, *flags, "-c", src, "-o", out]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
    elif src.endswith(".cpp"):
        cmd = [nvcc(), "-O2", "-std=c++17", "-Xcompiler", "-fPIC", *inc, "-c", src, "-o", out]
    else:
        cmd = ["gcc", "-O2", "-std=c11", "-fPIC", "-Wall", *inc, "-c", src, "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"compiling {src} failed:\n{r.stdout}\n{r.stderr}")
    return out, r.stderr


def build(verbose=False, force=False):
    srcs = [os.path.join(CSRC, s) for s in SOURCES]
    # every header of the library and of include/ is a dependency of every object
    deps = srcs + sorted(glob.glob(os.path.join(CSRC, "*.h")) + glob.glob(os.path.join(CSRC, "*.cuh")) +
                         glob.glob(os.path.join(REPO, "include", "*.h")))
    if not force and os.path.exists(LIB) and os.path.getmtime(LIB) >= max(os.path.getmtime(d) for d in deps):
        return LIB
    os.makedirs(BUILD, exist_ok=True)
    units = []
    for src in srcs:
        name = os.path.basename(src)
        for tag, t in PARTS.get(name, []):
            units.append((src, f"{name}.{tag}", [f"-DUKG_NAME={tag}", f"-DUKG_TYPE={t}"] + (SPLIT if tag == "f64" else [])))
        units.append((src, name, SPLIT if src.endswith(".cu") and name not in WHOLE else []))
    with cf.ThreadPoolExecutor(max_workers=len(units)) as ex:
        results = list(ex.map(lambda u: _compile(u, verbose), units))
    if verbose:
        for _, err in results:
            if err:
                sys.stderr.write(err)
    objs = [o for o, _ in results]
    cmd = [nvcc(), *ARCH, "-shared", "-o", LIB + ".tmp", *objs, "-lcudart_static", "-lrt", "-ldl", "-lpthread"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"linking libukgpu.so failed:\n{r.stdout}\n{r.stderr}")
    os.replace(LIB + ".tmp", LIB)
    return LIB


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv, force=True))
