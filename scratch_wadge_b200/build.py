"""Build recipe of the CUDA library libwadg_b200.so (sm_100a, in-tree)."""

from __future__ import annotations

import glob
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
LIB = os.path.join(HERE, "libwadg_b200.so")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
# uncompressed device code: nvcc compresses what is over some 10 MB, and a degree's first
# kernel in a process then takes 8-12 ms to unpack its object instead of 5-6 to load it
COMPRESS = ["-compress-mode=none"]


def sources():
    return sorted(glob.glob(os.path.join(HERE, "csrc", "*.cu")) +
                  glob.glob(os.path.join(HERE, "csrc", "*.cpp")))


def deps():
    return sources() + sorted(glob.glob(os.path.join(HERE, "csrc", "*.cuh"))) + \
        [os.path.join(ROOT, "include", "wadg.h"), __file__]


def build(force=False, verbose=False, extra=()):
    if not force and os.path.exists(LIB) and \
            all(os.path.getmtime(d) <= os.path.getmtime(LIB) for d in deps()):
        return LIB
    objs = []
    bdir = os.path.join(HERE, "_build")
    os.makedirs(bdir, exist_ok=True)
    procs = []
    for src in sources():
        obj = os.path.join(bdir, os.path.basename(src) + ".o")
        cmd = [NVCC, "-O3", "-std=c++17", *ARCH, *COMPRESS, "-lineinfo", "-Xcompiler", "-fPIC",
               "-Xptxas", "-v" if verbose else "-O3", "-I", os.path.join(ROOT, "include"),
               "-c", src, "-o", obj, *extra]
        procs.append((cmd, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    for cmd, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0:
            raise RuntimeError("nvcc failed: " + " ".join(cmd) + "\n" + out)
        if verbose:
            print(out)
    cmd = [NVCC, "-shared", *ARCH, "-o", LIB, *objs, "-lcudart_static", "-lrt", "-ldl", "-lpthread"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("link failed: " + " ".join(cmd) + "\n" + r.stdout + r.stderr)
    return LIB


if __name__ == "__main__":
    import sys
    print(build(force=True, verbose="-v" in sys.argv))
