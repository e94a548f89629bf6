"""Builds libmustafar_b200.so (all CUDA sources of csrc/, sm_100a only) and, where the interpreter's C headers are
installed, _native.<ABI tag>.so (the CPython binding of its hot entry points) in-tree with nvcc.

    python -m mustafar_b200.build [--force] [--verbose]

nvcc cross-compiles without a GPU.  Objects are rebuilt only when a source or
header is newer; the shared library sits next to this file so that it travels
with the source tree.
"""
from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libmustafar_b200.so")
# the tag keeps a tree built for one interpreter from loading its binding into another
NATIVE = os.path.join(HERE, "_native" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so"))
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
FLAGS = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC=/path/to/nvcc")


def _newest_header() -> float:
    t = os.path.getmtime(os.path.join(os.path.dirname(HERE), "include", "mustafar_b200.h"))
    for f in os.listdir(CSRC):
        if f.endswith((".cuh", ".h")):
            t = max(t, os.path.getmtime(os.path.join(CSRC, f)))
    return t


def build_native(nvcc: str, hdr_t: float, force: bool = False) -> str | None:
    """The binding is a shortcut, not a requirement: without Python.h it is left out and the package calls the same
    functions through ctypes."""
    include = sysconfig.get_path("include")
    if not os.path.exists(os.path.join(include, "Python.h")):
        sys.stderr.write(f"no Python.h in {include}: the CPython binding is left out\n")
        return None
    src = os.path.join(CSRC, "native.cpp")
    if force or not os.path.exists(NATIVE) or os.path.getmtime(NATIVE) < max(os.path.getmtime(src), hdr_t):
        cmd = [nvcc, "-O2", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-cudart", "none", "-o", NATIVE, src,
               "-I", include, "-L", HERE, "-l:" + os.path.basename(LIB), "-Xlinker", "-rpath=$ORIGIN"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
            raise RuntimeError("the CPython binding failed to build")
    return NATIVE


def build(force: bool = False, verbose: bool = False) -> str:
    nvcc = _nvcc()
    os.makedirs(OBJ, exist_ok=True)
    srcs = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))
    hdr_t = _newest_header()
    flags = list(FLAGS)
    if verbose:
        flags = flags + ["-Xptxas", "-v"]
    jobs = []
    for f in srcs:
        src = os.path.join(CSRC, f)
        obj = os.path.join(OBJ, f[:-3] + ".o")
        if force or not os.path.exists(obj) or os.path.getmtime(obj) < max(os.path.getmtime(src), hdr_t):
            jobs.append((src, obj))

    def run(job):
        src, obj = job
        cmd = [nvcc, *ARCH, *flags, "-c", src, "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        return cmd, r

    with ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as ex:
        for cmd, r in ex.map(run, jobs):
            if verbose or r.returncode != 0:
                sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
            if r.returncode != 0:
                raise RuntimeError("nvcc failed for " + cmd[-3])
    objs = [os.path.join(OBJ, f[:-3] + ".o") for f in srcs]
    if jobs or not os.path.exists(LIB):
        cmd = [nvcc, *ARCH, "-shared", "-o", LIB, *objs, "-lcudart"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link failed")
    build_native(nvcc, hdr_t, force)
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose))
