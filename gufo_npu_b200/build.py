"""Builds libgufo_cuda.so (the C-ABI library, nvcc for sm_100a) and the extension module _native (the
Python side's per-call work, the host compiler) in-tree."""
from __future__ import annotations

import importlib.util
import os
import runpy
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libgufo_cuda.so")
NATIVE = os.path.join(HERE, "_native" + sysconfig.get_config_var("EXT_SUFFIX"))   # of this interpreter

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
]


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _stale(target: str = LIB, suffixes=(".cu", ".cuh")) -> bool:
    if not os.path.exists(target):
        return True
    built = os.path.getmtime(target)
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(suffixes)]
    return any(os.path.getmtime(d) > built for d in deps + [os.path.join(ROOT, "include", "gufo_cuda.h")])


def build_native(force: bool = False) -> str:
    """Compiles csrc/native.cpp against the interpreter's and torch's headers; returns its path."""
    torch = os.path.dirname(importlib.util.find_spec("torch").origin)
    version = runpy.run_path(os.path.join(torch, "version.py"))["__version__"]
    if not force and not _stale(NATIVE, (".cpp",)):
        with open(NATIVE, "rb") as f:
            if version.encode() + b"\0" in f.read():   # built for this torch
                return NATIVE
    untagged = os.path.join(HERE, "_native.so")
    if os.path.exists(untagged):   # any interpreter would take it
        os.remove(untagged)
    include = os.path.join(torch, "include")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-Wall", "-fvisibility=hidden",
           f'-DGUFO_TORCH_VERSION="{version}"',
           "-I", os.path.join(ROOT, "include"), "-I", sysconfig.get_paths()["include"], "-isystem", include,
           "-isystem", os.path.join(include, "torch", "csrc", "api", "include"), "-isystem", "/usr/local/cuda/include",
           os.path.join(CSRC, "native.cpp"), "-o", NATIVE,
           "-L", os.path.join(torch, "lib"), "-ltorch_python", "-ltorch_cpu", "-lc10", "-ldl"]
    subprocess.run(cmd, check=True)
    return NATIVE


def build(force: bool = False, verbose: bool = False) -> str:
    """Compiles every .cu under csrc/ into one shared library; returns its path. The Python
    extension is built beside it."""
    build_native(force)
    if not force and not _stale():
        return LIB
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    extra = os.environ.get("GUFO_NVCC_EXTRA", "").split()   # e.g. -DGUFO_STEP_DEBUG_STAMPS for a timing probe
    objs = []
    for src in sources():
        obj = os.path.join(CSRC, os.path.basename(src)[:-3] + ".o")
        cmd = [nvcc, *NVCC_FLAGS, *extra, "-I", os.path.join(ROOT, "include"), "-I", CSRC, "-c", src, "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
            print(" ".join(cmd), file=sys.stderr)
        subprocess.run(cmd, check=True)
        objs.append(obj)
    cmd = [nvcc, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a"]
    subprocess.run(cmd, check=True)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
