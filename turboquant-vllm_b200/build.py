"""Build libtq4_sm100a.so (the C-ABI CUDA library) and _tq4_host.*.so (its CPython binding) in-tree.

Usage:  python turboquant-vllm_b200/build.py [--force] [--verbose]
Both land in turboquant-vllm_b200/turboquant_vllm/lib/.  The CUDA library is compiled with nvcc for
sm_100a and has a plain C ABI (include/tq4.h, no torch headers); the binding (csrc/tq4_host.cpp) is
compiled with g++ against the headers of the installed torch and links to it.  Its name carries the
Python ABI and the torch version it was built for, as the package looks for it: after a change of
either, the old binary is neither loaded nor taken for up to date.
"""
from __future__ import annotations

import argparse
import glob
import importlib.metadata
import importlib.util
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
OUT_DIR = os.path.join(HERE, "turboquant_vllm", "lib")
OUT = os.path.join(OUT_DIR, "libtq4_sm100a.so")
HOST_SRC = os.path.join(CSRC, "tq4_host.cpp")



def host_name() -> str:
    """File name of the CPython binding for this interpreter and the installed torch."""
    return f"_tq4_host.{sysconfig.get_config_var('SOABI')}.torch{importlib.metadata.version('torch')}.so"


HOST_OUT = os.path.join(OUT_DIR, host_name())


def sources() -> list[str]:
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _deps() -> list[str]:
    return glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.h")) + [
        os.path.join(ROOT, "include", "tq4.h")]


def needs_build() -> bool:
    if not os.path.exists(OUT) or host_needs_build():
        return True
    t = os.path.getmtime(OUT)
    return any(os.path.getmtime(d) > t for d in sources() + _deps())


def host_needs_build() -> bool:
    if not os.path.exists(HOST_OUT):
        return True
    t = os.path.getmtime(HOST_OUT)
    return any(os.path.getmtime(d) > t for d in (HOST_SRC, os.path.join(ROOT, "include", "tq4.h")))


def host_command() -> list[str]:
    """g++ command line of the CPython binding (linked to the CUDA library beside it)."""
    torch_dir = os.path.dirname(importlib.util.find_spec("torch").origin)
    inc = os.path.join(torch_dir, "include")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    return [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", "-o", HOST_OUT, HOST_SRC,
            "-I", inc, "-I", os.path.join(inc, "torch", "csrc", "api", "include"), "-I", os.path.join(cuda, "include"),
            "-I", sysconfig.get_paths()["include"], "-I", os.path.join(ROOT, "include"),
            "-L", os.path.join(torch_dir, "lib"), "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda",
            "-L", OUT_DIR, "-l:libtq4_sm100a.so", "-Wl,-rpath,$ORIGIN"]


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu to an object file (in parallel, only those older than their inputs) and
    link the shared library."""
    if not force and not needs_build():
        return OUT
    os.makedirs(OUT_DIR, exist_ok=True)
    obj_dir = os.path.join(HERE, "build")
    os.makedirs(obj_dir, exist_ok=True)
    nvcc = os.environ.get("NVCC", "nvcc")
    flags = ["-Xcompiler", "-fPIC", "-O3", "-std=c++17", "-lineinfo",
             "-gencode", "arch=compute_100a,code=sm_100a",
             "-I", os.path.join(ROOT, "include"), "-I", CSRC]
    if verbose:
        flags += ["-Xptxas", "-v"]
    hdr_time = max(os.path.getmtime(d) for d in _deps())
    jobs, objs = [], []
    for src in sources():
        obj = os.path.join(obj_dir, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        stale = force or verbose or not os.path.exists(obj) or os.path.getmtime(obj) < max(
            os.path.getmtime(src), hdr_time)
        if stale:
            jobs.append((src, subprocess.Popen([nvcc, "-c", *flags, "-o", obj, src])))
    failed = [src for src, p in jobs if p.wait() != 0]
    if failed:
        raise subprocess.CalledProcessError(1, f"nvcc -c {' '.join(failed)}")
    if jobs or not os.path.exists(OUT):
        subprocess.run([nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", OUT, *objs], check=True)
    else:
        os.utime(OUT)
    if force or host_needs_build():
        subprocess.run(host_command(), check=True)
    return OUT


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose))
