"""Build recipe of the CUDA extension: one shared library, sm_103a only.

Compiles each translation unit with nvcc in parallel and links
`libavbd_gb300.so` in-tree (next to this file). The geometry units
(narrowphase, broadphase) are built with --fmad=false so their f64
arithmetic matches the reference engine operation for operation.
"""
from __future__ import annotations

import concurrent.futures as cf
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
BUILD = os.path.join(HERE, "_build")
LIB = os.path.join(HERE, "libavbd_gb300.so")
ARCH = ["-gencode", "arch=compute_103a,code=sm_103a"]
# A unit's image is read whole when a process first needs any of it; compressed (the default for images as large as
# the solver's), that made the first pack of a process 15 ms instead of 3.5.
PLAIN_IMAGE = ["--compress-mode=none"]
UNITS = {
    "narrowphase.cu": ["--fmad=false"],
    "broadphase.cu": ["--fmad=false"],
    "solver.cu": [],
    "host.cu": [],
    "tangent.cu": ["--fmad=false"],
    "repack.cu": [],
}


def nvcc():
    for cand in (shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def _stale(out, deps):
    if not os.path.exists(out):
        return True
    t = os.path.getmtime(out)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False, ptxas_verbose: bool = False) -> str:
    os.makedirs(BUILD, exist_ok=True)
    headers = [os.path.join(CSRC, h) for h in ("avbd_device.cuh", "collider.cuh", "dual.cuh")]
    headers.append(os.path.join(HERE, "..", "include", "avbd_cuda.h"))
    objs = []
    jobs = []
    for unit, extra in UNITS.items():
        src = os.path.join(CSRC, unit)
        obj = os.path.join(BUILD, unit.replace(".cu", ".o"))
        objs.append(obj)
        if force or _stale(obj, [src] + headers):
            cmd = [nvcc(), *ARCH, *PLAIN_IMAGE, "-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC", "-rdc=false",
                   "-c", src, "-o", obj, *extra]
            if ptxas_verbose:
                cmd += ["-Xptxas", "-v"]
            jobs.append(cmd)
    with cf.ThreadPoolExecutor(max_workers=len(UNITS)) as ex:
        for cmd, res in zip(jobs, ex.map(lambda c: subprocess.run(c, capture_output=True, text=True), jobs)):
            if verbose or res.returncode != 0 or ptxas_verbose:
                sys.stderr.write(res.stdout + res.stderr)
            if res.returncode != 0:
                raise RuntimeError("nvcc failed: " + " ".join(cmd))
    if force or jobs or not os.path.exists(LIB):
        cmd = [nvcc(), *ARCH, "-shared", "-o", LIB, *objs, "-lcudart", "-lpthread"]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            sys.stderr.write(res.stdout + res.stderr)
            raise RuntimeError("link failed")
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose=True, ptxas_verbose="-v" in sys.argv)
    print(LIB)
