"""Ahead-of-time build of the native library (no JIT at run time).

``python -m fleet_chiplet_megakernel_b200._build`` or ``build()`` compiles the
CUDA sources for sm_100a into ``libb200mk.so`` next to this file.  The built
library is what the package loads; there is no fallback when it is missing.
"""
import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libb200mk.so")
# mk_kernel_tp.cu, mk_kernel_hier.cu and mk_kernel_moe.cu include mk_kernel.cu with other build switches (see its header); each
# is compiled once per linear path (MK_NC, see mk_launch.cu)
SOURCES = {"mk_kernel.cu": (0, 8, 16, 32), "mk_kernel_tp.cu": (0, 8, 16, 32), "mk_kernel_hier.cu": (0, 8, 16, 32), "mk_kernel_moe.cu": (0, 8),
           "mk_launch.cu": None, "mk_runtime.cpp": None, "mk_noalloc.cu": None}
HEADERS = ["mk_types.h", "mk_wide.cuh", os.path.join("..", "..", "include", "b200mk.h")]


def _nvcc():
    for c in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if c and os.path.exists(c):
            return c
    raise RuntimeError("nvcc not found: the native library cannot be built")


def needs_build():
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = [os.path.join(CSRC, s) for s in list(SOURCES) + HEADERS]
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def build(force=False, verbose=False):
    if not force and not needs_build():
        return LIB
    flags = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC"]
    if verbose:
        flags = ["-Xptxas", "-v"] + flags
    objdir = os.path.join(HERE, "build")
    os.makedirs(objdir, exist_ok=True)
    jobs = []
    for src, instances in SOURCES.items():
        stem = os.path.splitext(src)[0]
        for nc in instances or (None,):
            obj = os.path.join(objdir, stem + ("" if nc is None else f"_{nc}") + ".o")
            define = [] if nc is None else [f"-DMK_NC={nc}"]
            jobs.append(([_nvcc()] + flags + define + ["-c", os.path.join(CSRC, src), "-o", obj], obj))
    # one nvcc per object, as many side by side as there are cores, then one link
    with ThreadPoolExecutor(max_workers=os.cpu_count() or 4) as pool:
        done = list(pool.map(lambda job: subprocess.run(job[0], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True), jobs))
    for (cmd, _), r in zip(jobs, done):
        if verbose or r.returncode != 0:
            sys.stdout.write(" ".join(cmd) + "\n" + r.stdout)
        if r.returncode != 0:
            raise subprocess.CalledProcessError(r.returncode, cmd)
    objs = [obj for _, obj in jobs]
    subprocess.check_call([_nvcc(), "-shared", "-o", LIB] + objs)
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose=True)
    print(LIB)
