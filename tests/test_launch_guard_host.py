"""Picking the kernel instance of a launch, on the CPU: mk_launch.cu over a CUDA runtime of a few recording functions."""
import ctypes as C
import json
import os
import subprocess

import pytest

from fleet_chiplet_megakernel_b200 import _build

FAKE = r"""
#include <cuda_runtime_api.h>
#include <string.h>
#include "mk_types.h"
static char insts[16];
static int regs[16], asked, launched;
#define INST(name, i) extern "C" const void* mk_instance_##name() { return insts + i; }
INST(base_0, 0) INST(base_8, 1) INST(base_16, 2) INST(base_32, 3) INST(tp_0, 4) INST(tp_8, 5) INST(tp_16, 6) INST(tp_32, 7)
INST(hier_0, 8) INST(hier_8, 9) INST(hier_16, 10) INST(hier_32, 11) INST(moe_0, 12)
static int index_of(const void* k) { return k >= insts && k < insts + 16 ? (int)((const char*)k - insts) : -1; }
extern "C" {
int mk_kernel_max_ctas_per_sm(const mk::KParams*, int);
int mk_kernel_max_clusters(const mk::KParams*, int, int, int);
int mk_kernel_launch(const mk::KParams*, int, int, void*);
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void* k) {
  if (index_of(k) < 0) return cudaErrorInvalidDeviceFunction;
  memset(a, 0, sizeof(*a));
  a->numRegs = regs[index_of(k)];
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* k, cudaFuncAttribute, int) { return index_of(k) < 0 ? cudaErrorInvalidDeviceFunction : cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void* k, int, size_t) { asked = index_of(k); *n = 1; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void* k, const cudaLaunchConfig_t*) { asked = index_of(k); *n = 37; return cudaSuccess; }
cudaError_t cudaLaunchCooperativeKernel(const void* k, dim3, dim3, void**, size_t, cudaStream_t) { launched = index_of(k); return cudaSuccess; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void* k, void**) { launched = index_of(k); return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t __cudaLaunchKernel_ptsz(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t __cudaGetKernel(cudaKernel_t*, const void*) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
void** __cudaRegisterFatBinary(void*) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
char __cudaInitModule(void**) { return 1; }
// out: what was asked about residency per SM, per cluster, what was launched (instance, or -1); ret: the three results
void probe(int few, int moe, int cluster, int world, int rows, int x_rows, int* out, int* ret) {
  for (int i = 0; i < 16; ++i) regs[i] = i == few ? mk::kLaunchRegs - 8 : mk::kLaunchRegs;
  static mk::KParams p;
  memset(&p, 0, sizeof(p));
  p.has_moe = moe; p.cluster = cluster; p.world = world; p.path = rows ? mk::PATH_ROWS : mk::PATH_WIDE; p.x_rows = x_rows;
  asked = launched = -1; ret[0] = mk_kernel_max_ctas_per_sm(&p, 1024); out[0] = asked;
  asked = -1; ret[1] = mk_kernel_max_clusters(&p, 1024, cluster, 148); out[1] = asked;
  ret[2] = mk_kernel_launch(&p, 148, 1024, nullptr); out[2] = launched;
}
}
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    d = tmp_path_factory.mktemp("launch")
    (d / "fake.cpp").write_text(FAKE)
    nvcc = _build._nvcc()
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-fPIC", "-I" + inc, "-I" + _build.CSRC, "-c", str(d / "fake.cpp"), "-o", str(d / "fake.o")])
    subprocess.check_call([nvcc, "-O1", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC", "-c",
                           os.path.join(_build.CSRC, "mk_launch.cu"), "-o", str(d / "launch.o")])

    def load(n):  # (a library of its own per case: an instance is asked about once per process)
        so = str(d / f"fake{n}.so")
        subprocess.check_call(["g++", "-shared", "-Wl,-Bsymbolic", "-o", so, str(d / "launch.o"), str(d / "fake.o")])
        return C.CDLL(so, mode=os.RTLD_LOCAL)
    return load


# the launch (MoE layers, CTAs per cluster, ranks, row-owner path, token rows of a box) and the instance that it runs
LAUNCHES = [((0, 1, 1, 1, 0), 0), ((0, 1, 1, 0, 16), 1), ((0, 1, 1, 0, 32), 2), ((0, 1, 1, 0, 64), 3), ((0, 1, 1, 0, 128), 3), ((0, 1, 2, 1, 0), 4),
            ((0, 1, 2, 0, 16), 5), ((0, 1, 2, 0, 32), 6), ((0, 1, 2, 0, 128), 7), ((0, 2, 1, 1, 0), 8), ((0, 4, 1, 0, 16), 9), ((0, 2, 1, 0, 32), 10),
            ((0, 2, 1, 0, 64), 11), ((1, 1, 1, 1, 0), 12), ((1, 2, 1, 1, 0), 12)]


@pytest.mark.parametrize("launch,inst", LAUNCHES)
def test_an_instance_with_too_few_registers_is_not_launched(fake, launch, inst):
    """The warp roles split the registers that a block is launched with; taking more than there are waits for good.  Every
    question about a launch is asked of the instance that runs, and the answer is no where its registers do not suffice."""
    out, ret = (C.c_int * 3)(), (C.c_int * 3)()
    lib = fake(f"{inst}_{launch[1]}_{launch[4]}_few")
    lib.probe(inst, *launch, out, ret)
    assert list(out) == [-1, -1, -1] and ret[0] == -1 and ret[1] == -1 and ret[2] != 0
    lib = fake(f"{inst}_{launch[1]}_{launch[4]}_enough")
    lib.probe(-1, *launch, out, ret)
    assert out[0] == inst and out[2] == inst and ret[0] == 1 and ret[1] == 37 and ret[2] == 0
    assert out[1] == inst or launch[1] == 1


def test_a_launch_without_an_instance_is_an_error(fake):
    """Mixture-of-experts programs serve one or two tokens: there is no instance of the wide path."""
    out, ret = (C.c_int * 3)(), (C.c_int * 3)()
    for x_rows in (16, 32, 64, 128):
        fake(f"none{x_rows}").probe(-1, 1, 1, 1, 0, x_rows, out, ret)
        assert list(out) == [-1, -1, -1] and ret[0] == -1 and ret[2] != 0


PTXAS = """ptxas info    : 0 bytes gmem
ptxas info    : Compiling entry function '_ZN2mk4base10megakernelILi1ELi8EEEvNS_7KParamsE' for 'sm_100a'
ptxas info    : Function properties for _ZN2mk4base10megakernelILi1ELi8EEEvNS_7KParamsE
    40 bytes stack frame, 120 bytes spill stores, 304 bytes spill loads
ptxas info    : Used 160 registers, used 16 barriers, 40 bytes cumulative stack size, 1024 bytes smem
ptxas info    : Compiling entry function '_ZN2mk17init_state_kernelENS_7KParamsE' for 'sm_100a'
ptxas info    : Function properties for _ZN2mk17init_state_kernelENS_7KParamsE
    0 bytes stack frame, 0 bytes spill stores, 0 bytes spill loads
ptxas info    : Used 26 registers, used 0 barriers
"""


def test_the_build_refuses_an_instance_with_too_few_registers():
    r = _build.resources(PTXAS)
    assert r == {"registers": 160, "stack": 40, "spill_stores": 120, "spill_loads": 304}
    assert _build.resources(PTXAS[PTXAS.index("init_state") - 60:]) is None
    with pytest.raises(RuntimeError, match="mk_kernel_8"):
        _build.check_registers({"mk_kernel_8": r, "mk_kernel_16": dict(r, registers=168)})
    with pytest.raises(RuntimeError, match="mk_kernel_8"):
        _build.check_registers({"mk_kernel_8": None})
    _build.check_registers({"mk_kernel_16": dict(r, registers=168)})


def test_every_built_instance_has_the_registers_of_the_split_and_no_spills(native_lib):
    if not os.path.exists(_build.REPORT):
        pytest.skip("the library was built elsewhere")
    with open(_build.REPORT) as f:
        built = json.load(f)
    assert set(built) == {f"{os.path.splitext(src)[0]}_{nc}" for src, ncs in _build.SOURCES.items() for nc in ncs or ()}
    _build.check_registers(built)
    # the two that gather the ranks' words in their epilogues or while they stage rows spill some of them; no other instance has
    # local memory
    assert {name for name, r in built.items() if r["stack"] or r["spill_stores"]} <= {"mk_kernel_tp_0", "mk_kernel_tp_32"}
