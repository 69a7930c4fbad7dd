"""Build libsnac_b200.so in-tree with nvcc for sm_100a.

    python -m snac_b200.build          # rebuild if a source changed
    python -m snac_b200.build --force

The CUDA files are compiled side by side, one nvcc each, with -fmad=false so
that every kernel rounds like the reference's x86-64 build (see
csrc/snac_device.cuh).  Which kernels share a file decides what their calls
cost in registers (csrc/snac_launch.cuh); no file is split among threads
(-split-compile), whose grouping, and with it the code, differs from one
build to the next.
"""
from __future__ import annotations

import glob
import os
import shutil
import subprocess
import sys
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libsnac_b200.so")
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]


def nvcc() -> str:
    for cand in (shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")) +
                  glob.glob(os.path.join(CSRC, "*.h")) +
                  [os.path.join(ROOT, "include", "snac_gpu.h")])


def stale() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    return any(os.path.getmtime(s) > t for s in sources())


def compile_commands(into: str, verbose: bool = False, defines=()):
    """One nvcc command for each CUDA file, its object in the folder `into`."""
    flags = [*ARCH, *["-D" + d for d in defines], "-lineinfo", "-O3", "-fmad=false", "-std=c++17",
             "-Xcompiler", "-fPIC,-O2", "-I" + os.path.join(ROOT, "include")]
    if verbose:
        flags.insert(0, "-Xptxas=-v")
    return [[nvcc(), *flags, "-c", "-o", os.path.join(into, os.path.basename(cu) + ".o"), cu]
            for cu in sorted(glob.glob(os.path.join(CSRC, "*.cu")))]


def build(force: bool = False, verbose: bool = False, defines=(), out: str = LIB) -> str:
    if not force and not stale() and out == LIB:
        return LIB
    with tempfile.TemporaryDirectory() as tmp:
        commands = compile_commands(tmp, verbose, defines)
        if verbose:
            print("\n".join(" ".join(c) for c in commands), flush=True)
        compilers = [subprocess.Popen(c) for c in commands]
        failed = [c for c, p in zip(commands, compilers) if p.wait() != 0]
        if failed:
            raise subprocess.CalledProcessError(1, failed[0])
        objects = [c[c.index("-o") + 1] for c in commands]
        subprocess.run([nvcc(), *ARCH, "-shared", "-o", out + ".tmp", *objects], check=True)
    os.replace(out + ".tmp", out)
    return out


def ensure_built() -> str:
    return build(force=False)


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(LIB)
