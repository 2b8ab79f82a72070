"""Builds libxn_mm.so (the C-ABI engine) in-tree with nvcc for sm_100a, and _host.so, the CPython module that is the
native host path of the Python operators.

    python xn_b200/build.py [--force] [--verbose]

The library links only the CUDA runtime; it has no Python or torch dependency.  The host module links the library
(found beside it at run time) and torch.
"""
from __future__ import annotations

import glob
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libxn_mm.so")
HOST_SRC = os.path.join(CSRC, "host", "binding.cpp")
HOST_LIB = os.path.join(HERE, "_host.so")
OBJ_DIR = os.path.join(HERE, "build")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-Wall", "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    for c in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if c and (os.path.isabs(c) and os.path.exists(c) or not os.path.isabs(c)):
            return c
    return "nvcc"


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def _torch_dir() -> str:
    import importlib.util
    return os.path.dirname(importlib.util.find_spec("torch").origin)  # without importing it


def _host_command() -> list[str]:
    t = _torch_dir()
    cuda = os.path.dirname(os.path.dirname(_nvcc())) if os.path.isabs(_nvcc()) else "/usr/local/cuda"
    return [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-Wall", "-fvisibility=hidden",
            "-D_GLIBCXX_USE_CXX11_ABI=1", "-isystem", os.path.join(t, "include"), "-isystem", os.path.join(cuda, "include"),
            "-isystem", sysconfig.get_paths()["include"], HOST_SRC, "-o", HOST_LIB, "-L" + HERE, "-l:libxn_mm.so", "-L" + os.path.join(t, "lib"),
            "-ltorch_python", "-ltorch_cpu", "-ltorch_cuda", "-lc10_cuda", "-lc10", "-Wl,-rpath,$ORIGIN"]


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ_DIR, exist_ok=True)
    headers = glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(HERE, "..", "include", "*.h"))
    objs, procs = [], []
    for src in sources():
        obj = os.path.join(OBJ_DIR, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        if force or _stale(obj, [src] + headers):
            cmd = [_nvcc(), *NVCC_FLAGS, "-c", src, "-o", obj]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
                print(" ".join(cmd), file=sys.stderr)
            procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0 or verbose:
            sys.stderr.write(out)
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed")
    if force or procs or _stale(LIB, objs):
        cmd = [_nvcc(), "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a", "-lcuda"]
        subprocess.check_call(cmd)
    # the module sees the library through the C ABI only: rebuilt when its source or the header changes
    if force or _stale(HOST_LIB, [HOST_SRC] + glob.glob(os.path.join(HERE, "..", "include", "*.h"))):
        cmd = _host_command()
        if verbose:
            print(" ".join(cmd), file=sys.stderr)
        subprocess.check_call(cmd)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
