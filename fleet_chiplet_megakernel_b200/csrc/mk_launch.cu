// Launching the megakernel: picks the instance of the kernel a program runs, and the kernel that resets the scheduler state.
#include <cuda_runtime.h>

#include <atomic>

#include "mk_types.h"

// mk_kernel.cu is compiled once per build (see its header) and per linear path: the row-owner path (0), and the wide path
// with 8, 16 or 32 token columns per finishing thread (half the rows of an activation box, at most 32).  Each is a module of its own, so
// that a process loads the one it runs.
#define MK_DECLARE(v) \
  extern "C" const void* mk_instance_##v##_0(); \
  extern "C" const void* mk_instance_##v##_8(); \
  extern "C" const void* mk_instance_##v##_16(); \
  extern "C" const void* mk_instance_##v##_32();
MK_DECLARE(base) MK_DECLARE(tp) MK_DECLARE(hier)
#undef MK_DECLARE
extern "C" const void* mk_instance_moe_0();

namespace mk {
__global__ void init_state_kernel(KParams p) {
  const int tid = threadIdx.x + blockIdx.x * blockDim.x;
  const int nth = blockDim.x * gridDim.x;
  for (int i = tid; i < p.total_requests; i += nth) p.step[i] = 0;
  for (int i = tid; i < p.max_reqs; i += nth) p.request_ids[i] = -1;
  for (int i = tid; i <= p.max_reqs; i += nth) {
    p.qo_indptr[i] = 0;
    p.kv_indptr[i] = 0;
  }
  for (int i = tid; i < p.max_pages; i += nth) p.page_queue[i] = i;
  if (tid == 0) {
    p.sched[0] = 0;
    p.sched[1] = p.max_pages;
    p.sched[2] = 0;
    p.sched[3] = 0;
    p.sched[4] = 0;
    p.sched[5] = 0;
    p.sched[6] = 0;
    p.sched[7] = 0;
  }
}
}  // namespace mk

namespace {
enum Build { BASE, TP, HIER, MOE };
using Instance = const void* (*)();
const Instance kInstances[4][4] = {
    {mk_instance_base_0, mk_instance_base_8, mk_instance_base_16, mk_instance_base_32},
    {mk_instance_tp_0, mk_instance_tp_8, mk_instance_tp_16, mk_instance_tp_32},
    {mk_instance_hier_0, mk_instance_hier_8, mk_instance_hier_16, mk_instance_hier_32},
    {mk_instance_moe_0, nullptr, nullptr, nullptr},  // (MoE layers are planned for one or two tokens only: row-owner path)
};
// The kernel that a launch with these parameters runs: tensor-parallel exchange code only when there are peers, the
// hierarchical barrier only when the launch uses clusters, the MoE ops only when the program has them.  Null where there is no
// such instance, or where it has fewer registers than the warp roles split among them: its setmaxnreg.inc would wait for good,
// the one wait of the kernel that nothing bounds.  (What an instance was compiled to does not change: asked once per process.)
const void* kernel_for(const mk::KParams* p, int cluster) {
  static std::atomic<int> fits[4][4];  // 0 not asked yet, 1 yes, -1 no
  const Build b = p->has_moe ? MOE : (cluster > 1 ? HIER : (p->world > 1 ? TP : BASE));
  const int i = p->path == mk::PATH_ROWS ? 0 : (p->x_rows <= 16 ? 1 : (p->x_rows <= 32 ? 2 : 3));
  if (!kInstances[b][i]) return nullptr;
  const void* k = kInstances[b][i]();
  int ok = fits[b][i].load(std::memory_order_relaxed);
  if (ok == 0) {
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, k) != cudaSuccess) return nullptr;  // (no device, or not this one: asked again)
    ok = fa.numRegs >= mk::kLaunchRegs ? 1 : -1;
    fits[b][i].store(ok, std::memory_order_relaxed);
  }
  return ok > 0 ? k : nullptr;
}
}  // namespace

extern "C" int mk_kernel_max_ctas_per_sm(const mk::KParams* p, int smem_bytes) {
  int n = 0;
  const void* k = kernel_for(p, p->cluster);
  if (!k || cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes) != cudaSuccess) return -1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, mk::kNumThreads, smem_bytes) != cudaSuccess) return -1;
  return n;
}

// Clusters of `cluster` CTAs that can be resident at once (the hierarchical barrier needs all of them).
extern "C" int mk_kernel_max_clusters(const mk::KParams* p, int smem_bytes, int cluster, int grid) {
  const void* k = kernel_for(p, cluster);
  if (!k || cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes) != cudaSuccess) return -1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(mk::kNumThreads);
  cfg.dynamicSmemBytes = (size_t)smem_bytes;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cluster;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  return n;
}

extern "C" int mk_kernel_launch(const mk::KParams* p, int grid, int smem_bytes, void* stream) {
  const void* k = kernel_for(p, p->cluster);
  if (!k) return (int)cudaErrorInvalidDeviceFunction;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
  if (e != cudaSuccess) return (int)e;
  void* args[] = {(void*)p};
  if (p->cluster <= 1) {
    e = cudaLaunchCooperativeKernel(k, dim3(grid), dim3(mk::kNumThreads), args, (size_t)smem_bytes, (cudaStream_t)stream);
    return (int)e;
  }
  // co-resident grid of thread-block clusters
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(mk::kNumThreads);
  cfg.dynamicSmemBytes = (size_t)smem_bytes;
  cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = p->cluster;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeCooperative;
  at[1].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  e = cudaLaunchKernelExC(&cfg, k, args);
  return (int)e;
}

extern "C" int mk_kernel_init_state(const mk::KParams* p, void* stream) {
  mk::init_state_kernel<<<4, 256, 0, (cudaStream_t)stream>>>(*p);
  return (int)cudaGetLastError();
}
