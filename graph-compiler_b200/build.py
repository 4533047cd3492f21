"""Build libGcDnnlApi.so (sm_100a) and its Python call path in-tree.

    python graph-compiler_b200/build.py [--force] [--verbose]

Every .cu/.cpp under csrc/ is compiled to an object with
``nvcc -gencode arch=compute_100a,code=sm_100a -lineinfo`` (objects are rebuilt
only when a source or header is newer) and linked into
``graph-compiler_b200/lib/libGcDnnlApi.so``; binding/gcb200_host.cpp (plain CPython API) becomes
``lib/_gcb200_host.so``.  nvcc cross-compiles, so this works
on a machine without a GPU.
"""
from __future__ import annotations

import argparse
import concurrent.futures as cf
import glob
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIBDIR = os.path.join(HERE, "lib")
LIB = os.path.join(LIBDIR, "libGcDnnlApi.so")
HOST = os.path.join(LIBDIR, "_gcb200_host.so")

NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
COMMON = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC,-fvisibility=hidden,-Wall", "-I", os.path.join(HERE, "..", "include")]


def _newest_header() -> float:
    hs = glob.glob(os.path.join(SRC, "*.h")) + glob.glob(os.path.join(SRC, "*.cuh")) + glob.glob(
        os.path.join(HERE, "..", "include", "*.h"))
    return max(os.path.getmtime(h) for h in hs) if hs else 0.0


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    os.makedirs(LIBDIR, exist_ok=True)
    srcs = sorted(glob.glob(os.path.join(SRC, "*.cu")) + glob.glob(os.path.join(SRC, "*.cpp")))
    hdr = _newest_header()
    jobs = []
    objs = []
    for s in srcs:
        o = os.path.join(OBJ, os.path.basename(s) + ".o")
        objs.append(o)
        if force or not os.path.exists(o) or os.path.getmtime(o) < max(os.path.getmtime(s), hdr):
            cmd = [NVCC, *ARCH, *COMMON, "-c", s, "-o", o]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        return cmd, r

    with cf.ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as ex:
        for cmd, r in ex.map(run, jobs):
            if verbose or r.returncode != 0:
                sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
            if r.returncode != 0:
                raise RuntimeError("nvcc failed for " + cmd[-3])
    if jobs or force or not os.path.exists(LIB):
        # link beside the target and rename: a reader (a running process, a copy of the tree) never sees a partial file
        tmp = LIB + ".tmp"
        link = [NVCC, *ARCH, "-shared", "-o", tmp, *objs, "-cudart", "static", "-Xlinker", "--no-undefined", "-lpthread", "-ldl", "-lrt"]
        r = subprocess.run(link, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link failed")
        os.replace(tmp, LIB)
    src = os.path.join(HERE, "binding", "gcb200_host.cpp")
    if force or not os.path.exists(HOST) or os.path.getmtime(HOST) < max(os.path.getmtime(src), hdr):
        tmp = HOST + ".tmp"
        cmd = ["g++", "-O2", "-std=c++17", "-Wall", "-shared", "-fPIC", "-fvisibility=hidden", "-I", sysconfig.get_paths()["include"], src,
               "-o", tmp, "-L", LIBDIR, "-lGcDnnlApi", "-Wl,-rpath,$ORIGIN"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("the Python binding did not build")
        os.replace(tmp, HOST)
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose))
