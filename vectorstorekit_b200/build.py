"""Builds ``libvsk_cuda.so`` (the C-ABI library) in-tree with nvcc for sm_100a.

    python -m vectorstorekit_b200.build            # build if sources are newer than the library
    python -m vectorstorekit_b200.build --force

nvcc cross-compiles without a GPU.  Object files go to ``vectorstorekit_b200/_build``.
"""
from __future__ import annotations

import concurrent.futures
import glob
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "_build")
LIB = os.path.join(HERE, "libvsk_cuda.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _deps_mtime() -> float:
    files = sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(HERE, "..", "include", "*.h"))
    return max(os.path.getmtime(f) for f in files)


def up_to_date(lib: str = LIB) -> bool:
    return os.path.exists(lib) and os.path.getmtime(lib) >= _deps_mtime()


def _build(lib: str, obj_dir: str, defines, force: bool, verbose: bool) -> str:
    if not force and up_to_date(lib):
        return lib
    os.makedirs(obj_dir, exist_ok=True)
    nvcc = _nvcc()
    hdr_mtime = max(os.path.getmtime(f) for f in glob.glob(os.path.join(CSRC, "*.cuh")) +
                    glob.glob(os.path.join(HERE, "..", "include", "*.h")))

    def compile_one(src):
        obj = os.path.join(obj_dir, os.path.basename(src)[:-3] + ".o")
        if (not force and os.path.exists(obj) and os.path.getmtime(obj) >= os.path.getmtime(src)
                and os.path.getmtime(obj) >= hdr_mtime):
            return obj, ""
        cmd = [nvcc] + NVCC_FLAGS + defines + (["-Xptxas", "-v"] if verbose else []) + ["-c", src, "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
        return obj, r.stderr

    with concurrent.futures.ThreadPoolExecutor(max_workers=8) as ex:
        results = list(ex.map(compile_one, sources()))
    if verbose:
        for _, log in results:
            sys.stderr.write(log)
    objs = [o for o, _ in results]
    # NCCL is looked up with dlopen when a communicator is first asked for: no -lnccl here
    cmd = [nvcc, "-shared", "-cudart", "static", "-o", lib] + objs + ["-lpthread", "-ldl"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    return lib


def build_library(force: bool = False, verbose: bool = False) -> str:
    return _build(LIB, OBJ, [], force, verbose)


# ---- the checked variant ---------------------------------------------------------------------------------------
LIB_CHECKED = os.path.join(HERE, "libvsk_cuda_checked.so")
OBJ_CHECKED = os.path.join(HERE, "_build_checked")


def build_checked(force: bool = False, verbose: bool = False) -> str:
    """``libvsk_cuda_checked.so``: the same sources with -DVSK_CHECKED, in which the kernels' read-only loads and atomics
    go through a range test (``csrc/checked.cuh``).  A testing aid; loaded with VSK_CHECKED=1."""
    return _build(LIB_CHECKED, OBJ_CHECKED, ["-DVSK_CHECKED"], force, verbose)


if __name__ == "__main__":
    if "--checked" in sys.argv:
        print(build_checked(force="--force" in sys.argv, verbose="-v" in sys.argv))
    else:
        print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
