"""Builds the CUDA library ``libmbr.so`` in-tree for sm_100a.

Every translation unit is compiled by nvcc with
``-gencode arch=compute_100a,code=sm_100a -lineinfo``; the strict FP64 unit is
compiled with ``--fmad=false`` so that its double arithmetic is the IEEE
sequence of the reference's CPU code.  Objects go to ``_build/``; a unit is
rebuilt when it or any header is newer than its object.

Usage: ``python -m mandelbulber2_b200.build [--force] [--jobs N]``.
"""
from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
BUILD = os.path.join(HERE, "_build")
LIB = os.path.join(HERE, "libmbr.so")

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
COMMON = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC", "-I", INCLUDE, "-I", CSRC]

# (source, extra flags)
UNITS = [
    ("mbr_host.cpp", []),
    ("fract_loader.cpp", []),
    ("plain_fp64.cu", []),
    ("plain_fp64_strict.cu", ["--fmad=false"]),
    ("staged_fp64.cu", []),
    ("staged_fp64_strict.cu", ["--fmad=false"]),
    ("staged_keyed_fp64.cu", []),
    ("staged_keyed_fp64_strict.cu", ["--fmad=false"]),
    ("plain_mixed.cu", []),
    ("wavefront.cu", []),
    ("wavefront32.cu", []),
    ("wavefront64.cu", []),
    ("wavefront_batch.cu", []),
    ("wavefront_hybrid.cu", []),
    ("probe.cu", []),
    ("adjoint.cu", []),
]


def nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", shutil.which("nvcc")):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def _headers() -> list[str]:
    hs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".h", ".cuh"))]
    hs.append(os.path.join(INCLUDE, "mbr.h"))
    return hs


def _stale(src: str, obj: str, headers: list[str]) -> bool:
    if not os.path.exists(obj):
        return True
    t = os.path.getmtime(obj)
    return any(os.path.getmtime(p) > t for p in [src, *headers])


def _compile(src: str, extra: list[str], force: bool, headers: list[str], verbose: bool) -> str:
    path = os.path.join(CSRC, src)
    obj = os.path.join(BUILD, os.path.splitext(src)[0] + ".o")
    if force or _stale(path, obj, headers):
        cmd = [nvcc(), *ARCH, *COMMON, *extra, "-c", path, "-o", obj]
        if src.endswith(".cu"):
            cmd += ["-Xptxas", "-v"] if verbose else []
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src}:\n{res.stderr}")
        if verbose and res.stderr:
            sys.stderr.write(res.stderr)
    return obj


def build(force: bool = False, jobs: int | None = None, verbose: bool = False) -> str:
    os.makedirs(BUILD, exist_ok=True)
    headers = _headers()
    jobs = jobs or min(len(UNITS), os.cpu_count() or 4)
    with ThreadPoolExecutor(max_workers=jobs) as ex:
        objs = list(ex.map(lambda u: _compile(u[0], u[1], force, headers, verbose), UNITS))
    if force or not os.path.exists(LIB) or any(os.path.getmtime(o) > os.path.getmtime(LIB) for o in objs):
        tmp = LIB + ".tmp"
        cmd = [nvcc(), *ARCH, "-shared", "-o", tmp, *objs, "-lcudart"]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"link failed:\n{res.stderr}")
        os.replace(tmp, LIB)
    return LIB


def main() -> None:
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--jobs", type=int, default=None)
    ap.add_argument("-v", "--verbose", action="store_true")
    a = ap.parse_args()
    print(build(force=a.force, jobs=a.jobs, verbose=a.verbose))


if __name__ == "__main__":
    main()
