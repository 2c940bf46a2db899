"""Ahead-of-time build of the native library (no JIT at run time).

``python -m fleet_chiplet_megakernel_b200._build`` or ``build()`` compiles the
CUDA sources for sm_100a into ``libb200mk.so`` next to this file.  The built
library is what the package loads; there is no fallback when it is missing.
"""
import json
import os
import re
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libb200mk.so")
OBJDIR = os.path.join(HERE, "build")
REPORT = os.path.join(OBJDIR, "instances.json")  # what ptxas made of every kernel instance
# mk_kernel_tp.cu, mk_kernel_hier.cu and mk_kernel_moe.cu include mk_kernel.cu with other build switches (see its header); each
# is compiled once per linear path that its programs take (MK_NC, see mk_launch.cu)
SOURCES = {"mk_kernel.cu": (0, 8, 16, 32), "mk_kernel_tp.cu": (0, 8, 16, 32), "mk_kernel_hier.cu": (0, 8, 16, 32), "mk_kernel_moe.cu": (0,),
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


def resources(ptxas):
    """Registers, stack and spills (bytes) a thread of the megakernel, from the output of ``ptxas -v``; None without one."""
    entry = re.search(r"Compiling entry function '\w*megakernel\w*'.*?(?=Compiling entry function|\Z)", ptxas, re.S)
    if entry is None:
        return None
    stack, stores, loads = map(int, re.search(r"(\d+) bytes stack frame, (\d+) bytes spill stores, (\d+) bytes spill loads", entry[0]).groups())
    return {"registers": int(re.search(r"Used (\d+) registers", entry[0])[1]), "stack": stack, "spill_stores": stores, "spill_loads": loads}


def check_registers(instances):
    """The warp roles share out kLaunchRegs registers a thread (mk_types.h): an instance with fewer would wait for them for good."""
    with open(os.path.join(CSRC, "mk_types.h")) as f:
        need = int(re.search(r"kLaunchRegs = (\d+)", f.read())[1])
    few = {name: r and r["registers"] for name, r in instances.items() if r is None or r["registers"] < need}  # (None: no kernel found)
    if few:
        raise RuntimeError(f"kernel instances with fewer than {need} registers a thread: {few}")


def build(force=False, verbose=False):
    if not force and not needs_build():
        return LIB
    flags = ["-Xptxas", "-v", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC"]
    os.makedirs(OBJDIR, exist_ok=True)
    jobs = []
    for src, instances in SOURCES.items():
        stem = os.path.splitext(src)[0]
        for nc in instances or (None,):
            obj = os.path.join(OBJDIR, stem + ("" if nc is None else f"_{nc}") + ".o")
            define = [] if nc is None else [f"-DMK_NC={nc}"]
            jobs.append(([_nvcc()] + flags + define + ["-c", os.path.join(CSRC, src), "-o", obj], obj))
    # one nvcc per object, as many side by side as there are cores, then one link
    with ThreadPoolExecutor(max_workers=os.cpu_count() or 4) as pool:
        done = list(pool.map(lambda job: subprocess.run(job[0], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True), jobs))
    instances = {}
    for (cmd, obj), r in zip(jobs, done):
        if verbose or r.returncode != 0:
            sys.stdout.write(" ".join(cmd) + "\n" + r.stdout)
        if r.returncode != 0:
            raise subprocess.CalledProcessError(r.returncode, cmd)
        name = os.path.splitext(os.path.basename(obj))[0]
        if name.startswith("mk_kernel"):
            instances[name] = resources(r.stdout)
    check_registers(instances)
    with open(REPORT, "w") as f:
        json.dump(instances, f, indent=1)
    objs = [obj for _, obj in jobs]
    subprocess.check_call([_nvcc(), "-shared", "-o", LIB] + objs)
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose=True)
    print(LIB)
