"""Builds libleviathan_cuda.so in-tree with nvcc for sm_100a.

Run as `python -m leviathan_b200.build`; `__graft_entry__.build()` calls
`build_library()`.  The shared library is linked with the static CUDA runtime
so it loads in any process without depending on another package's libcudart.
"""
from __future__ import annotations

import glob
import os
import subprocess
import sys
import sysconfig
from importlib.machinery import EXTENSION_SUFFIXES

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libleviathan_cuda.so")
HOST_PATH = os.path.join(LIB_DIR, "_pyhost" + EXTENSION_SUFFIXES[0])

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-lineinfo", "-std=c++17",
    "-Xcompiler", "-fPIC,-Wall,-Wno-unused-function",
    "-cudart", "static",
    "-I", os.path.join(ROOT, "include"),
    "-I", CSRC,
]


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build_library(force: bool = False, verbose: bool = False) -> str:
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    os.makedirs(LIB_DIR, exist_ok=True)
    obj_dir = os.path.join(HERE, "build")
    os.makedirs(obj_dir, exist_ok=True)
    sources = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    headers = sorted(glob.glob(os.path.join(CSRC, "*.h")) + glob.glob(os.path.join(CSRC, "*.cuh"))
                     + glob.glob(os.path.join(ROOT, "include", "*.h")))
    objects = []
    procs = []
    for src in sources:
        obj = os.path.join(obj_dir, os.path.basename(src)[:-3] + ".o")
        objects.append(obj)
        if force or _stale(obj, [src] + headers):
            cmd = [nvcc, *NVCC_FLAGS, *os.environ.get("LEV_NVCC_EXTRA", "").split(), "-c", src, "-o", obj]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if out.strip():
            print(out, file=sys.stderr)
        if p.returncode != 0:
            failed = True
            print(f"nvcc failed on {src}", file=sys.stderr)
    if failed:
        raise RuntimeError("libleviathan_cuda.so: compilation failed")
    if force or procs or _stale(LIB_PATH, objects):
        cmd = [nvcc, "-shared", "-cudart", "static", "-gencode", "arch=compute_100a,code=sm_100a",
               "-o", LIB_PATH, *objects, "-ldl", "-lpthread"]
        subprocess.run(cmd, check=True)
    # The native calls of the Python layer (csrc/lev_pyhost.c) for this interpreter, bound to the library beside them.
    # Without a C compiler or Python's headers the package goes through ctypes.
    src = os.path.join(CSRC, "lev_pyhost.c")
    if force or _stale(HOST_PATH, [src, LIB_PATH] + headers):
        cmd = [os.environ.get("CC", "gcc"), "-O2", "-Wall", "-shared", "-fPIC", "-I", os.path.join(ROOT, "include"),
               "-I", sysconfig.get_paths()["include"], "-o", HOST_PATH, src, "-L", LIB_DIR, "-l:libleviathan_cuda.so", "-Wl,-rpath,$ORIGIN"]
        try:
            subprocess.run(cmd, check=True)
        except (OSError, subprocess.CalledProcessError) as e:
            if os.path.exists(HOST_PATH):
                os.remove(HOST_PATH)
            print(f"lev_pyhost.c is not built ({e}): calls go through ctypes", file=sys.stderr)
    return LIB_PATH


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
