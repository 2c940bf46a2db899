// The persistent decode megakernel for sm_100a.
//
// One cooperative launch runs a whole generation.  Every SM hosts one CTA: warp 8 is a TMA
// producer that streams this CTA's share of every linear layer's weights (boxes of 64 k-elements,
// 128-byte swizzle) into a ring of shared-memory stages, running ahead of the consumers across op
// boundaries (weights have no dependencies); the eight consumer warps walk the program: wait at a
// grid barrier where an op reads what other CTAs wrote, do the op's share of work, go on.  Warp 10 issues the
// linears' tcgen05 instructions; the wide path (mk_wide.cuh) has two more roles, an activation producer and a norm warp.  Every wait in
// the kernel is bounded: on expiry the waiter records a status and raises a sticky abort flag that
// all other waits poll, and the kernel returns with an error code.
//
// Replaces the worker/scheduler loops of the reference runtime
// (include/mirage/persistent_kernel/persistent_kernel.cuh:693-1854) and its
// task kernels (tasks/blackwell/*.cuh, tasks/ampere/*.cuh, tasks/hopper/rmsnorm_hopper.cuh).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "mk_types.h"

// This file is compiled several times into one library (see the wrappers mk_kernel_tp.cu,
// mk_kernel_hier.cu and mk_kernel_moe.cu, and mk_launch.cu): the persistent kernel runs every op body
// once per layer, and code that is merely present in an op (a branch for another configuration, the
// registers it pins) measurably slows a step down.  So the single-GPU kernels carry no tensor-parallel
// exchange code (+2.8 % when present), only the kernels launched in thread-block clusters carry the
// hierarchical grid barrier (+2.0 %), and each instance holds one linear path.
//
// There are no calls in an instance: with one, its per-thread context lives in local memory, calls save
// and restore registers there, and the register split of the warp roles (consumer_regs) has no effect.
// A block then had 200 to 320 KB of local memory beside an L1 of 28 to 92 KB.  Without calls it has
// none (but for 88 and 16 bytes a thread in the tensor-parallel instances for one or two and for 33 to 128 tokens).  Measured
// against the same code with out-of-line functions, 12 layers of 8B width, us per step: one request 1283 -> 1109, two
// 1468 -> 1166, eight of 300 tokens 1707 -> 1477, 32 of 100 1878 -> 1588, 64 of 100 2340 -> 1942; four layers 1024 wide, one
// request 172 -> 134.
//   MK_NC             linear path: 0 the row-owner path, 8, 16 or 32 the wide path (token columns of a finishing thread)
//   MK_VARIANT        inner namespace of this compilation: base | tp | hier | moe
//   MK_WITH_XCHG      1: linear epilogues can push to / input staging can gather from the ranks' exchange regions
//   MK_HIER_BARRIER   1: cluster-first grid barrier (the kernel must be launched with a cluster dimension)
//   MK_WITH_MOE       1: the mixture-of-experts ops (routing, per-expert row-owner linears, weighted combine)
#ifndef MK_NC
#define MK_NC 0
#endif
#ifndef MK_VARIANT
#define MK_VARIANT base
#endif
#ifndef MK_WITH_XCHG
#define MK_WITH_XCHG 0
#endif
#ifndef MK_HIER_BARRIER
#define MK_HIER_BARRIER 0
#endif
#ifndef MK_WITH_MOE
#define MK_WITH_MOE 0
#endif
#if MK_WITH_XCHG
#define MK_XF(op, f) ((op).flags & (f))
#else
#define MK_XF(op, f) 0
#endif

namespace mk {
namespace MK_VARIANT {

// ------------------------------------------------------------------------------------
// PTX helpers
// ------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ unsigned long long globaltimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_n(uint32_t bar, uint32_t n) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(n) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Asks once, without the suspension of try_wait: for a thread that watches several barriers.
__device__ __forceinline__ bool mbar_test_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// The same, suspended for no longer than about `ns`.
__device__ __forceinline__ bool mbar_try_wait_for(uint32_t bar, uint32_t parity, uint32_t ns) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(ns)
      : "memory");
  return ok != 0;
}
// 2-D tiled TMA load into this CTA only: box {64 k-elements, 128 rows} at (x = k, y = row).
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const void* tmap, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(tmap), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
// The same with an L2 eviction policy (from createpolicy) attached to the lines it reads.
__device__ __forceinline__ void tma_load_2d_hint(uint32_t dst, const void* tmap, uint32_t bar, int x, int y, uint64_t pol) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4}], [%2], %5;"
      ::"r"(dst), "l"(tmap), "r"(bar), "r"(x), "r"(y), "l"(pol)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_hint(uint32_t dst, const void* tmap, uint32_t bar, int x, int y, int z, uint64_t pol) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4, %5}], [%2], %6;" ::"r"(dst),
      "l"(tmap), "r"(bar), "r"(x), "r"(y), "r"(z), "l"(pol)
      : "memory");
}
__device__ __forceinline__ void tma_prefetch_2d(const void* tmap, int x, int y) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(tmap), "r"(x), "r"(y) : "memory");
}
// One lane of a converged warp.
__device__ __forceinline__ bool elect_one() {
  uint32_t is;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(is));
  return is != 0u;
}
// ---- tcgen05: descriptors, completion, shared memory -> tensor memory
__device__ __forceinline__ uint64_t umma_smem_desc(uint32_t saddr, uint32_t group_bytes = 1024u) {
  // start address >> 4 | leading offset (unused for swizzled K-major) 1 | stride between 8-row
  // groups >> 4 | descriptor version 1 | layout 2 = 128-byte swizzle
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | (1ull << 16) | ((uint64_t)(group_bytes >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// the same with A in tensor memory: 16 k-elements of 128 rows are eight columns
__device__ __forceinline__ void umma_bf16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// 128 rows x 64 k-elements of a swizzled stage (16 KB) -> 128 lanes x 32 columns of tensor memory: lane = row, column c = k-elements 2 c
// and 2 c + 1.
__device__ __forceinline__ void tmem_put_128x64(uint32_t tmem, uint32_t saddr) {
  const uint64_t d = umma_smem_desc(saddr);
#pragma unroll
  for (int q = 0; q < 4; ++q)  // 16 k-elements = 32 bytes further inside the swizzle span
    asm volatile("tcgen05.cp.cta_group::1.128x256b [%0], %1;" ::"r"(tmem + 8u * q), "l"(d + (uint64_t)(2 * q)) : "memory");
}
// one accumulator column of this warp's 32 lanes; the caller waits with tmem_wait_ld
__device__ __forceinline__ uint32_t tmem_ld1(uint32_t taddr) {
  uint32_t r;
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(r) : "r"(taddr) : "memory");
  return r;
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void consumer_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
  return v;
}
__device__ __forceinline__ void sts128(uint32_t addr, const uint4& v) {
  asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
// barrier counter and abort flag (adjacent words) in one load
__device__ __forceinline__ uint2 ld_bar_pair(const unsigned* p) {
  uint2 v;
  asm volatile("ld.acquire.gpu.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ float bf_lo(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float bf_hi(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }
__device__ __forceinline__ void unpack8(const uint4& v, float* f) {
  f[0] = bf_lo(v.x); f[1] = bf_hi(v.x); f[2] = bf_lo(v.y); f[3] = bf_hi(v.y);
  f[4] = bf_lo(v.z); f[5] = bf_hi(v.z); f[6] = bf_lo(v.w); f[7] = bf_hi(v.w);
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ uint4 pack8(const float* f) {
  return make_uint4(pack2(f[0], f[1]), pack2(f[2], f[3]), pack2(f[4], f[5]), pack2(f[6], f[7]));
}
__device__ __forceinline__ float rbf(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// ------------------------------------------------------------------------------------
// per-thread context
// ------------------------------------------------------------------------------------
struct Ctx {
  const KParams& p;
  uint8_t* smem;
  uint32_t smem_addr;
  unsigned epoch;     // grid barriers passed
  bool arrived;       // this CTA has already arrived at the coming grid barrier
  int attn_iter;      // row-owner path: iteration whose attention metadata is cached in shared memory; wide path: head geometry planned
  uint32_t tmem;      // base address of the CTA's tensor-memory columns
  unsigned acc_runs;  // accumulator runs (row-owner path: chunks) finished
  int tid, lane, warp;
  int iter, cur_op;
  unsigned long long* dbg;  // inner-phase stamps of the traced op (thread 0), or null
  unsigned long long* pr;   // this op's trace record, or null
  bool dead;                // abort flag seen at the op's barrier (CTA-uniform)
  unsigned ar_seq;          // cross-rank exchanges (allreduce pushes) executed so far in this launch
  unsigned lin_seq;         // linear ops whose barrier has been passed in this launch
#if MK_HIER_BARRIER
  unsigned nbar;            // grid barriers waited for in this launch (phase of the cluster mbarriers)
  uint32_t cl_rank, cl_size;  // this CTA's rank in its thread-block cluster, CTAs per cluster
#endif
  __device__ Ctx(const KParams& p_) : p(p_) {}
  // Every op starts from values the compiler cannot trace to the kernel's start: else it works out what depends on the
  // thread's index for all ops ahead of the op loop, and spills it there.
  __device__ __forceinline__ void opaque() {
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid));
    lane = tid & 31;
    warp = tid >> 5;
    asm volatile("" : "+l"(smem), "+r"(smem_addr), "+r"(tmem));
  }
  // mbarriers, groups of kMaxStages: weights of a stage landed, and its shared memory free again; (wide path) activation boxes ready,
  // their memory free, the raw rows of a box that still has to be normalised; a slot of the
  // weight ring's part in tensor memory free again
  __device__ uint32_t bar_of(int group, int s) const { return smem_addr + p.bar_off + 8 * (group * kMaxStages + s); }
  __device__ uint32_t full_bar(int s) const { return bar_of(0, s); }
  __device__ uint32_t empty_bar(int s) const { return bar_of(1, s); }
  __device__ uint32_t xfull_bar(int s) const { return bar_of(2, s); }
  __device__ uint32_t xempty_bar(int s) const { return bar_of(3, s); }
  __device__ uint32_t xraw_bar(int s) const { return bar_of(4, s); }
  __device__ uint32_t tfree_bar(int s) const { return bar_of(5, s); }
  // wide path: the activation boxes of stage s, behind the weights of all stages
  __device__ uint32_t xbox(int s) const { return smem_addr + (uint32_t)(p.num_stages * kStageBytes + s * (p.stage_bytes - kStageBytes)); }
  __device__ volatile int* flags() const { return (volatile int*)(smem + p.bar_off + kFlagsOff); }
  // behind the flags: the end-of-work mbarrier of the tcgen05 issuer and the word tcgen05.alloc writes
  __device__ uint32_t done_bar() const { return smem_addr + p.bar_off + kFlagsOff + 64; }
  __device__ uint32_t tmem_slot() const { return smem_addr + p.bar_off + kFlagsOff + 72; }
  // hierarchical grid barrier: arrivals of the cluster (used in its first CTA), release from the first CTA, its abort word
  __device__ uint32_t cl_arrive_bar() const { return smem_addr + p.bar_off + kFlagsOff + 80; }
  __device__ uint32_t cl_open_bar() const { return smem_addr + p.bar_off + kFlagsOff + 88; }
  __device__ uint32_t cl_dead_word() const { return smem_addr + p.bar_off + kFlagsOff + 96; }
  // wide path, per accumulator buffer: sums complete (tcgen05.commit), sums fetched (one arrival per finishing warp)
  __device__ uint32_t acc_full_bar(unsigned b) const { return smem_addr + p.bar_off + kFlagsOff + 104 + 8 * b; }
  __device__ uint32_t acc_empty_bar(unsigned b) const { return smem_addr + p.bar_off + kFlagsOff + 120 + 8 * b; }
  __device__ float* sums() const { return (float*)(smem + p.sums_off); }
  __device__ float* red() const { return (float*)(smem + p.red_off); }  // small scratch: reductions, lengths
};
// flags(): [0] go word written by consumers, read by the producer
//          [1] stages issued by the producer   [2] broadcast slot   [3] dead flag of the op
//          [4] linear ops whose barrier the consumers have passed   [5] stages taken from the ring by the tcgen05 issuer
//          [6] wide path: linear ops whose row scales are in the token table

#define MK_STAMP(c, k)                                             \
  do {                                                            \
    if ((c).dbg != nullptr && (c).tid == 0) (c).dbg[k] = globaltimer(); \
  } while (0)

__device__ __forceinline__ void raise_abort_at(const KParams* p, int iter, int op, int code, int d0, int d1) {
  if (atomicCAS(p->abort_flag, 0, 1) == 0) {
    p->status[0] = code;
    p->status[1] = blockIdx.x;
    p->status[2] = op;
    p->status[3] = iter;
    p->status[4] = d0;
    p->status[5] = d1;
    p->status[6] = threadIdx.x;
    __threadfence();
  }
}
__device__ __forceinline__ void raise_abort(const Ctx& c, int code, int d0, int d1) {
  raise_abort_at(&c.p, c.iter, c.cur_op, code, d0, d1);
}
__device__ __forceinline__ bool aborted(const Ctx& c) { return *(volatile int*)c.p.abort_flag != 0; }

// Bounded wait on an mbarrier phase.  Returns false after raising the abort flag.
// The clock is only consulted every few thousand failed polls: reading %globaltimer
// is slow enough to throttle the weight stream if it sits on the per-tile path.
// Time limits are tiered so that the record names the root cause: a wait on another GPU gives
// up after timeout_ns, waits on other CTAs or on the producer after twice that, the producers'
// own waits (on the consumers) after four times.
__device__ __forceinline__ bool mbar_wait_slow(const KParams* p, int iter, int op, uint32_t bar, uint32_t parity, int code) {
  unsigned long long t0 = 0;
  unsigned polls = 0;
  while (true) {
    if (mbar_try_wait(bar, parity)) return true;
    if (((++polls) & 4095u) == 0) {
      if (*(volatile int*)p->abort_flag != 0) return false;
      const unsigned long long now = globaltimer();
      if (t0 == 0) {
        t0 = now;
      } else if (now - t0 > p->timeout_ns * (code == ST_TIMEOUT_EMPTY ? 4ull : 2ull)) {
        raise_abort_at(p, iter, op, code, (int)bar, (int)parity);
        return false;
      }
    }
  }
}
// Fast path: a few hundred polls without touching the clock; then the bounded slow path.
__device__ __forceinline__ bool mbar_wait(const Ctx& c, uint32_t bar, uint32_t parity, int code) {
#pragma unroll 1
  for (int i = 0; i < 256; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  return mbar_wait_slow(&c.p, c.iter, c.cur_op, bar, parity, code);
}

// The weight ring as its tcgen05 issuer sees it: stages in shared memory, and slots of tensor memory for tiles that have to wait
// for their activations.  Tiles are used in order, those in slots (the older ones) first.
//
// Weights depend on nobody, so between two ops the ring fills up and HBM would idle until the first activations are there: split
// sums, words or a barrier, staging, 4 to 18 us, of which three to four stages are 2 to 3.  So while there is nothing to multiply,
// the oldest stage goes into a slot (tcgen05.cp, 0.27 us) and is loaded again.  While there is, nothing goes into a slot: every tile
// through tensor memory streams at 1.16 us a tile instead of 0.69 (copies and products take turns on the same pipe), and mma.sync
// stands still while a copy is under way.  `flying`: loads that may still be under way when a stage goes into a slot, which is how
// hard the stream goes on while words are polled and barriers are waited for: it slows them down.  All of them on the row-owner
// path, one up to 32 token rows, none beyond.  12 layers of 8B width, us per step with none, one and all: one request 1057, 1032,
// 1010; 4 requests 1190, 1167, 1213; 8 1245, 1220, 1270; 32 1419, 1408, 1425; 64 1668, 1685, 1734; 100 2215, 2228, 2220; without
// slots: one request 1086, 8 1303, 64 1732.  With four slots instead of six one request takes 1031 instead of 1004.
//
// The issuer is an elected lane, not lane 0: behind elect.sync the compiler issues tcgen05 from uniform registers.  Eight products
// (128 x 16 x 16 each, the same up to 64 columns) and a commit take 400 cycles instead of 920, of the 1350 in which HBM delivers
// a tile; the step at 8 requests fell from 1392 to 1303 us with it.
struct WeightRing {
  const Ctx& c;
  const int S, slots;
  const uint32_t slot0;
  int s = 0;                         // next stage
  uint32_t parity = 0;
  int head = 0, tail = 0, held = 0;  // slots: the oldest tile, the next to fill, tiles held
  uint32_t tail_parity = 1;
  unsigned taken = 0;                // stages taken from the ring
  __device__ __forceinline__ WeightRing(const Ctx& c_, int slots_, uint32_t slot0_) : c(c_), S(c_.p.num_stages), slots(slots_), slot0(slot0_) {}
  __device__ __forceinline__ uint32_t stage() const { return c.smem_addr + (uint32_t)(s * kStageBytes); }
  __device__ __forceinline__ uint32_t slot() const { return slot0 + (uint32_t)(head * kSlotCols); }
  // what reads the next stage, or the oldest slot, has been issued
  __device__ __forceinline__ void free_stage() {
    umma_commit(c.empty_bar(s));
    ++taken;
    if (++s == S) {
      s = 0;
      parity ^= 1u;
    }
  }
  __device__ __forceinline__ void free_slot() {
    umma_commit(c.tfree_bar(head));
    if (++head == slots) head = 0;
    --held;
  }
  // the oldest stage goes into a slot, when there is one and all stages but the `flying` newest have landed (both ends are looked
  // at: copies may land out of order)
  __device__ __forceinline__ void set_aside(int flying) {
    const int last = s + S - 1 - flying, at = last >= S ? last - S : last;
    if (held == slots || !mbar_test_wait(c.full_bar(s), parity) || !mbar_test_wait(c.full_bar(at), last >= S ? parity ^ 1u : parity) ||
        !mbar_test_wait(c.tfree_bar(tail), tail_parity)) return;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t src = stage(), dst = slot0 + (uint32_t)(tail * kSlotCols);
    tmem_put_128x64(dst, src);
    tmem_put_128x64(dst + 32u, src + kSubBytes);
    ++held;
    if (++tail == slots) {
      tail = 0;
      tail_parity ^= 1u;
    }
    free_stage();
  }
  // a bounded wait that sets tiles aside meanwhile
  __device__ __forceinline__ bool wait(uint32_t bar, uint32_t par, int flying = 0) {
    unsigned long long since = 0;
    unsigned polls = 0;
    while (!mbar_try_wait_for(bar, par, 200u)) {
      set_aside(flying);
      if (((++polls) & 1023u) == 0) {
        if (aborted(c)) return false;
        const unsigned long long now = globaltimer();
        if (since == 0) {
          since = now;
        } else if (now - since > 4 * c.p.timeout_ns) {
          raise_abort(c, ST_TIMEOUT_FULL, (int)bar, (int)par);
          return false;
        }
      }
    }
    return true;
  }
  // a tile to multiply
  __device__ __forceinline__ bool wait_tile() { return held > 0 || mbar_wait(c, c.full_bar(s), parity, ST_TIMEOUT_FULL); }
};

// Grid-wide barrier of the consumer warps.  The counter only grows within a launch: barrier
// number e is passed when it reaches e * (arrivals per barrier), compared modulo 2^32 so
// that a long launch may wrap it.
//
// Two shapes, chosen by the host per launch (KParams::cluster):
//  * flat (cluster = 1): every CTA adds 1 to the counter in L2 and polls it.
//  * hierarchical (cluster = 2 or 4, the kernel is launched in thread-block clusters): the CTAs
//    of a cluster first meet on an mbarrier in the shared memory of the cluster's first CTA
//    (remote arrive over distributed shared memory, release at cluster scope); that CTA alone
//    adds 1 to the global counter, polls it, and then opens an mbarrier in each of its peers'
//    shared memory.  The global line sees gridDim.x / cluster arrivals and pollers instead of
//    gridDim.x.  (The reference's Fleet runtime counts arrivals per XCD before one global release
//    per XCD, persistent_kernel.cuh:1214-1275; this is the same idea on Blackwell's clusters.)
//
// The arrival half on its own: an op that has loads to issue which do not depend on other
// CTAs arrives first and issues them while the others catch up.
#if MK_HIER_BARRIER
__device__ __forceinline__ uint32_t cluster_map(uint32_t local_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait on an mbarrier that CTAs of the same cluster arrive on.
__device__ __forceinline__ bool cluster_bar_wait(const Ctx& c, uint32_t bar, uint32_t parity) {
  unsigned long long t0 = 0;
  unsigned polls = 0;
  while (true) {
    if (mbar_try_wait_cluster(bar, parity)) return true;
    if (((++polls) & 1023u) == 0) {
      if (aborted(c)) return false;
      const unsigned long long now = globaltimer();
      if (t0 == 0) {
        t0 = now;
      } else if (now - t0 > 2 * c.p.timeout_ns) {
        raise_abort(c, ST_TIMEOUT_GRID, (int)c.epoch, -(int)c.cl_rank - 1);
        return false;
      }
    }
  }
}
__device__ __forceinline__ void grid_arrive(Ctx& c) {
  consumer_sync();
  c.epoch += 1;
  c.arrived = true;
  if (c.tid == 0) {
    // arrive with a release: nothing comes back, polling can start at once
    if (c.cl_size == 1) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(c.p.grid_bar) : "memory");
    else mbar_arrive_cluster(cluster_map(c.cl_arrive_bar(), 0));
  }
}
// The waiting half: values loaded ahead of the barrier stay in registers across it.
__device__ __forceinline__ void grid_wait(Ctx& c) {
  c.arrived = false;
  if (c.tid == 0) {
    bool dead = false;
    if (c.cl_rank == 0) {
      if (c.cl_size > 1) {
        // the cluster is complete: one arrival for all of it (the release is cumulative over what
        // the peers published to this thread through the mbarrier)
        if (cluster_bar_wait(c, c.cl_arrive_bar(), c.nbar & 1u))
          asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(c.p.grid_bar) : "memory");
        else
          dead = true;
      }
      const unsigned target = c.epoch * (gridDim.x / c.cl_size);
      unsigned long long t0 = 0;
      unsigned spins = 0;
      // the abort flag is the word behind the counter: one 8-byte load polls both
      while (!dead) {
        const uint2 v = ld_bar_pair(c.p.grid_bar);
        if (v.y != 0u) {
          dead = true;
          break;
        }
        if ((int)(v.x - target) >= 0) break;
        if (((++spins) & 1023u) == 0) {
          const unsigned long long now = globaltimer();
          if (t0 == 0) {
            t0 = now;
          } else if (now - t0 > 2 * c.p.timeout_ns) {
            raise_abort(c, ST_TIMEOUT_GRID, (int)c.epoch, (int)ld_acquire_u32(c.p.grid_bar));
            dead = true;
            break;
          }
        }
      }
      for (uint32_t r = 1; r < c.cl_size; ++r) {
        asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], %1;" ::"r"(cluster_map(c.cl_dead_word(), r)), "r"(dead ? 1u : 0u) : "memory");
        mbar_arrive_cluster(cluster_map(c.cl_open_bar(), r));
      }
    } else {
      if (!cluster_bar_wait(c, c.cl_open_bar(), c.nbar & 1u)) dead = true;
      else dead = *reinterpret_cast<volatile uint32_t*>(c.smem + c.p.bar_off + kFlagsOff + 96) != 0u;
    }
    c.flags()[3] = dead ? 1 : 0;
  }
  c.nbar += 1;
  consumer_sync();
}
#else
__device__ __forceinline__ void grid_arrive(Ctx& c) {
  consumer_sync();
  c.epoch += 1;
  c.arrived = true;
  // arrive with a release reduction: nothing comes back, polling can start at once
  if (c.tid == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(c.p.grid_bar) : "memory");
}
// The waiting half: values loaded ahead of the barrier stay in registers across it.
__device__ __forceinline__ void grid_wait(Ctx& c) {
  c.arrived = false;
  if (c.tid == 0) {
    const unsigned target = c.epoch * gridDim.x;
    unsigned long long t0 = 0;
    unsigned spins = 0;
    // the abort flag is the word behind the counter: one 8-byte load polls both
    bool dead = false;
    while (true) {
      const uint2 v = ld_bar_pair(c.p.grid_bar);
      if (v.y != 0u) {
        dead = true;
        break;
      }
      if ((int)(v.x - target) >= 0) break;
      if (((++spins) & 1023u) == 0) {
        const unsigned long long now = globaltimer();
        if (t0 == 0) {
          t0 = now;
        } else if (now - t0 > 2 * c.p.timeout_ns) {
          raise_abort(c, ST_TIMEOUT_GRID, (int)c.epoch, (int)ld_acquire_u32(c.p.grid_bar));
          dead = true;
          break;
        }
      }
    }
    c.flags()[3] = dead ? 1 : 0;
  }
  consumer_sync();
}
#endif  // MK_HIER_BARRIER
__device__ __forceinline__ void grid_sync(Ctx& c) {
  if (!c.arrived) grid_arrive(c);
  grid_wait(c);
}

// Every op calls this once, after whatever it can fetch ahead of its dependencies:
// the grid barrier (if the op has one) and the CTA-uniform abort check.  Returns
// true when the abort flag is up and the op body must be skipped.
__device__ __forceinline__ bool op_barrier(Ctx& c, const OpDesc& op) {
  if (op.flags & F_SYNC_BEFORE) {
    grid_sync(c);
  } else {
    if (c.tid == 0) c.flags()[3] = aborted(c) ? 1 : 0;
    consumer_sync();
  }
  if (c.pr != nullptr && c.tid == 0) c.pr[1] = globaltimer();
  c.dead = c.flags()[3] != 0;
  return c.dead;
}

// ------------------------------------------------------------------------------------
// tensor-parallel exchange over NVLink peer memory (the two allreduces of a layer)
// ------------------------------------------------------------------------------------
// The reference's allreduce is an NVSHMEM put-with-signal allgather followed by a local
// reduction task (src/kernel/task_register.cc:1606-1687, tasks/ampere/reduction.cuh:139-166).
// Here every rank stores its fp32 partial sums straight into EVERY rank's exchange region
// (its own included) with plain stores over NVLink, as 8-byte words {value, exchange number}:
// a word that carries the awaited number has arrived, so no fence, flag or second round trip
// is needed, and a reader simply adds the ranks' words up in rank order in fp32 (identical
// on every rank) and rounds once to bf16.  Data always lands in the reader's own memory; no
// bulk or tensor copy ever touches a peer's memory.  The halves of a region alternate between
// consecutive exchanges: a rank can only push exchange s+2 after it has read all of s+1 from
// every peer, which those peers push after their last read of s.
// Words travel as what they are, 64-bit scalars {value, number}: only those are single-copy atomic.  (Of a vector of 32-bit scalars
// the memory model lets the number be newer than the value beside it.)
__device__ __forceinline__ uint4 ld_sys_words(const uint4* p) {
  uint4 v;
  asm volatile(
      "{\n\t.reg .b64 a, b;\n\tld.relaxed.sys.global.v2.b64 {a,b}, [%4];\n\tmov.b64 {%0,%1}, a;\n\tmov.b64 {%2,%3}, b;\n\t}"
      : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
      : "l"(p)
      : "memory");
  return v;
}
__device__ __forceinline__ uint2 ld_sys_word(const uint2* p) {
  uint2 v;
  asm volatile("{\n\t.reg .b64 a;\n\tld.relaxed.sys.global.b64 a, [%2];\n\tmov.b64 {%0,%1}, a;\n\t}" : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_sys_word(uint2* p, uint32_t value, uint32_t number) {
  asm volatile("{\n\t.reg .b64 a;\n\tmov.b64 a, {%1,%2};\n\tst.relaxed.sys.global.b64 [%0], a;\n\t}" ::"l"(p), "r"(value), "r"(number) : "memory");
}
// two words at once, of the same number
__device__ __forceinline__ void st_sys_words(uint4* p, uint32_t a, uint32_t b, uint32_t number) {
  asm volatile(
      "{\n\t.reg .b64 a, b;\n\tmov.b64 a, {%1,%3};\n\tmov.b64 b, {%2,%3};\n\tst.relaxed.sys.global.v2.b64 [%0], {a,b};\n\t}" ::"l"(p), "r"(a), "r"(b), "r"(number)
      : "memory");
}
// one value of exchange `seq` into every rank's region
__device__ __forceinline__ void xchg_push1(const KParams& p, unsigned seq, int tok, int col, float v) {
  const size_t w = xchg_word(seq, p.world, p.xchg_tokens, p.xchg_cols, p.rank, tok, col);
#pragma unroll 1
  for (int r = 0; r < p.world; ++r) st_sys_word(reinterpret_cast<uint2*>(p.xchg[r]) + w, __float_as_uint(v), seq);
}
// A word of a rank that is not there yet: poll it (bounded).  Returns false after raising the abort flag.
__device__ __forceinline__ bool xchg_wait_word(const Ctx& c, const uint2* w, unsigned seq, int src) {
  unsigned long long t0 = 0;
  unsigned spins = 0;
  while (true) {
    if (xchg_arrived(ld_sys_word(w).y, seq)) return true;
    if (((++spins) & 63u) == 0) {
      if (aborted(c)) return false;
      const unsigned long long now = globaltimer();
      if (t0 == 0) {
        t0 = now;
      } else if (now - t0 > c.p.timeout_ns) {
        raise_abort(c, ST_TIMEOUT_RANK, src, (int)seq);
        return false;
      }
    }
  }
}
// 8 consecutive columns (col a multiple of 8) of token row `tok`: the sum over ranks as bf16 x 8
__device__ __forceinline__ uint4 xchg_gather8(const Ctx& c, unsigned seq, int tok, int col) {
  const KParams& p = c.p;
  float acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;
#pragma unroll 1
  for (int r = 0; r < p.world; ++r) {
    const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const uint2*>(p.xchg[p.rank]) +
                                                      xchg_word(seq, p.world, p.xchg_tokens, p.xchg_cols, r, tok, col));
    uint4 q[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) q[i] = ld_sys_words(src + i);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (!xchg_arrived(q[i].y, seq) || !xchg_arrived(q[i].w, seq)) {
        const uint2* w2 = reinterpret_cast<const uint2*>(src + i);
        if (!xchg_wait_word(c, w2, seq, r) || !xchg_wait_word(c, w2 + 1, seq, r)) return make_uint4(0, 0, 0, 0);
        q[i] = ld_sys_words(src + i);
      }
      acc[2 * i] += __uint_as_float(q[i].x);
      acc[2 * i + 1] += __uint_as_float(q[i].z);
    }
  }
  return pack8(acc);
}
// one column: the bf16-rounded sum over ranks, as a float
__device__ __forceinline__ float xchg_gather1(const Ctx& c, unsigned seq, int tok, int col) {
  const KParams& p = c.p;
  float acc = 0.f;
#pragma unroll 1
  for (int r = 0; r < p.world; ++r) {
    const uint2* w = reinterpret_cast<const uint2*>(p.xchg[p.rank]) + xchg_word(seq, p.world, p.xchg_tokens, p.xchg_cols, r, tok, col);
    uint2 q = ld_sys_word(w);
    if (!xchg_arrived(q.y, seq)) {
      if (!xchg_wait_word(c, w, seq, r)) return 0.f;
      q = ld_sys_word(w);
    }
    acc += __uint_as_float(q.x);
  }
  return rbf(acc);
}
// number of the latest exchange (the one gathering ops read) and of the one a pushing linear writes
__device__ __forceinline__ unsigned xchg_cur(const Ctx& c) { return xchg_seq(c.p.xchg_seq_base, c.ar_seq); }
__device__ __forceinline__ unsigned xchg_next(const Ctx& c) { return xchg_seq(c.p.xchg_seq_base, c.ar_seq + 1u); }

// ------------------------------------------------------------------------------------
// Tagged activations between the ops of the row-owner path.  A producer stores every pair of adjacent
// bf16 outputs as one 8-byte word {pair, tag}; 8-byte stores are single-copy atomic, so a word that
// carries the awaited tag carries its data: the consumer needs no grid barrier, no fence and no second
// round trip, it simply polls the words it is going to read anyway.  Eight columns are four words,
// read as two 16-byte loads.
// ------------------------------------------------------------------------------------
__device__ __forceinline__ uint4 ld_gpu_words(const uint4* p) {
  uint4 v;
  asm volatile(
      "{\n\t.reg .b64 a, b;\n\tld.relaxed.gpu.global.v2.b64 {a,b}, [%4];\n\tmov.b64 {%0,%1}, a;\n\tmov.b64 {%2,%3}, b;\n\t}"
      : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
      : "l"(p)
      : "memory");
  return v;
}
__device__ __forceinline__ uint2 ld_gpu_word(const uint2* p) {
  uint2 v;
  asm volatile("{\n\t.reg .b64 a;\n\tld.relaxed.gpu.global.b64 a, [%2];\n\tmov.b64 {%0,%1}, a;\n\t}" : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_gpu_word(uint2* p, uint32_t value, uint32_t tag) {
  asm volatile("{\n\t.reg .b64 a;\n\tmov.b64 a, {%1,%2};\n\tst.relaxed.gpu.global.b64 [%0], a;\n\t}" ::"l"(p), "r"(value), "r"(tag) : "memory");
}
// two words at once, of the same number
__device__ __forceinline__ void st_gpu_words(uint4* p, uint32_t a, uint32_t b, uint32_t tag) {
  asm volatile(
      "{\n\t.reg .b64 a, b;\n\tmov.b64 a, {%1,%3};\n\tmov.b64 b, {%2,%3};\n\tst.relaxed.gpu.global.v2.b64 [%0], {a,b};\n\t}" ::"l"(p), "r"(a), "r"(b), "r"(tag)
      : "memory");
}
__device__ __forceinline__ bool ll_ok(const uint4& a, const uint4& b, unsigned tag) {
  return a.y == tag && a.w == tag && b.y == tag && b.w == tag;
}
// The bound of a poll: true (after raising the abort flag) when the wait has to end without its data.
struct PollLimit {
  unsigned spins = 0;
  unsigned long long t0 = 0;
  __device__ __forceinline__ bool expired(const Ctx& c, unsigned tag, unsigned got, int code = ST_TIMEOUT_DATA) {
    if (((++spins) & 63u) != 0) return false;
    if (aborted(c)) return true;
    const unsigned long long now = globaltimer();
    if (t0 == 0) {
      t0 = now;
    } else if (now - t0 > 2 * c.p.timeout_ns) {
      raise_abort(c, code, (int)tag, (int)got);
      return true;
    }
    return false;
  }
};
// N vectors of eight columns: vector i from src + 2 at[i] where at[i] >= 0, else zeros.  All loads first, then whatever
// has not arrived is loaded again, all of it per trip: one loop, where a poll per vector was as many copies of its code
// (inlined) or as many calls.
template <int N>
__device__ __forceinline__ void ll_take(const Ctx& c, const uint4* src, const int (&at)[N], unsigned tag, uint4 (&out)[N]) {
  uint4 a[N], b[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const unsigned t = at[i] >= 0 ? ~tag : tag;  // (nothing to wait for: zeros that carry the tag)
    a[i] = b[i] = make_uint4(0u, t, 0u, t);
  }
  PollLimit limit;
  while (true) {
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (!ll_ok(a[i], b[i], tag)) {
        a[i] = ld_gpu_words(src + 2 * at[i]);
        b[i] = ld_gpu_words(src + 2 * at[i] + 1);
      }
    bool here = true;
#pragma unroll
    for (int i = 0; i < N; ++i) here = here && ll_ok(a[i], b[i], tag);
    if (here || limit.expired(c, tag, a[0].y)) break;
  }
#pragma unroll
  for (int i = 0; i < N; ++i) out[i] = make_uint4(a[i].x, a[i].z, b[i].x, b[i].z);
}
// one column, as a float
__device__ __forceinline__ float ll_gather1(const Ctx& c, const uint2* row, int col, unsigned tag) {
  const uint2* w = row + (col >> 1);
  PollLimit limit;
  uint2 q;
  do q = ld_gpu_word(w);
  while (q.y != tag && !limit.expired(c, tag, q.y));
  return (col & 1) ? bf_hi(q.x) : bf_lo(q.x);
}
__device__ __forceinline__ const uint2* ll_row(const void* base, int ld, int tok) {
  return reinterpret_cast<const uint2*>(base) + (size_t)tok * (size_t)(ld >> 1);
}
// the tag of what program op `op` stores in the current iteration
__device__ __forceinline__ unsigned ll_tag_of(const Ctx& c, int op) { return ll_tag(c.iter, c.p.num_ops, op); }

#if MK_WITH_XCHG
// Tensor parallelism, row-owner path: the reader of an exchange does not add up all of it in every CTA
// (that is `world` dependent round trips per CTA and `world` times the row in loads).  Every CTA adds up
// its own slice of the columns, in rank order in fp32 with one bf16 rounding (the same value on every
// rank), and stores it as tagged words; all CTAs then stage the row from those words like any other
// tagged input: two round trips whatever the number of ranks.
__device__ __forceinline__ void xchg_reduce_slice(Ctx& c, const OpDesc& op, int T) {
  const KParams& p = c.p;
  const int pairs = op.k >> 1;
  const int p0 = (int)((long long)blockIdx.x * pairs / gridDim.x), p1 = (int)((long long)(blockIdx.x + 1) * pairs / gridDim.x);
  const int w = p1 - p0;
  const unsigned seq = xchg_cur(c);
  const unsigned tag = ll_tag_of(c, c.cur_op);
  uint2* dst = reinterpret_cast<uint2*>(const_cast<void*>(op.ll_in));
#pragma unroll 1
  for (int i = c.tid; i < w * T; i += kNumConsumers) {
    const int tok = i / w, pr = p0 + i % w;
    uint4 q[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      if (r < p.world)
        q[r] = ld_sys_words(reinterpret_cast<const uint4*>(reinterpret_cast<const uint2*>(p.xchg[p.rank]) +
                                                        xchg_word(seq, p.world, p.xchg_tokens, p.xchg_cols, r, tok, 2 * pr)));
    }
    float a0 = 0.f, a1 = 0.f;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      if (r < p.world) {
        if (!xchg_arrived(q[r].y, seq) || !xchg_arrived(q[r].w, seq)) {
          const uint2* w2 = reinterpret_cast<const uint2*>(p.xchg[p.rank]) + xchg_word(seq, p.world, p.xchg_tokens, p.xchg_cols, r, tok, 2 * pr);
          if (!xchg_wait_word(c, w2, seq, r) || !xchg_wait_word(c, w2 + 1, seq, r)) return;
          q[r] = ld_sys_words(reinterpret_cast<const uint4*>(w2));
        }
        a0 += __uint_as_float(q[r].x);
        a1 += __uint_as_float(q[r].z);
      }
    }
    st_gpu_word(dst + (size_t)tok * (size_t)(op.ld_in >> 1) + pr, pack2(a0, a1), tag);
  }
}
#endif

// ------------------------------------------------------------------------------------
__device__ __forceinline__ float torch_rsqrt_bf16(float var, bool dbl);

// activations -> shared memory, with the optional fused RMSNorm
// ------------------------------------------------------------------------------------
// Row-owner path: token rows as the tensor core reads them (see linear_pass_rows), a row every x_pitch(kp) vectors of 16 bytes, kp
// a multiple of 512 there: the 64 vectors of a 512-wide k stage are eight rows (the stage's 64-wide slices) of 128 bytes,
// 128-byte swizzled.  Wide path (rows gathered from the ranks only): plain rows.
__device__ __forceinline__ int x_pitch(int kp) { return kp >> 3; }
__device__ __forceinline__ int x_vec(int v) { return MK_NC == 0 ? v ^ ((v >> 3) & 7) : v; }
// Stage `rows` (at most 8) token rows (tokens tok0.. of T; absent ones zero) of a K-wide
// bf16 input in shared memory, RMS-normalised when norm_w is given.  All
// rows are staged concurrently: the 8 consumer warps split into one group per row (8 warps
// on a single row, 1 warp per row for 5 to 8 rows), a group's warps take interleaved
// 512-byte pieces of the row and meet once to add up their sums of squares.  The loops are
// kept rolled on purpose: this runs once per op, straight from a cold instruction cache.
//
// `pre_w`: when not null, this lane's first 4 norm-weight vectors (vector index
// part * 32 + lane + 32 * wpr * i), loaded by the caller ahead of the op's barrier; rows of
// at most 4 vectors per lane then stay in registers between the two passes.
__device__ __forceinline__ int stage_warps_per_row(int rows) { return rows <= 1 ? 8 : (rows == 2 ? 4 : (rows <= 4 ? 2 : 1)); }

// sum of squares of 8 bf16 values; `torch_num`: each square rounded to bf16 first
__device__ __forceinline__ float sumsq8(const uint4& val, bool torch_num, float ss) {
  float f[8];
  unpack8(val, f);
  if (torch_num) {
#pragma unroll
    for (int i = 0; i < 8; ++i) ss += rbf(f[i] * f[i]);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) ss += f[i] * f[i];
  }
  return ss;
}
// 8 values scaled by r and the norm weight: w * bf16(x * r), or x * (r * w) in fp32
__device__ __forceinline__ uint4 scale8(const uint4& val, const uint4& wvec, float r, bool torch_num) {
  float f[8], w[8];
  unpack8(val, f);
  unpack8(wvec, w);
  if (torch_num) {
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = w[i] * rbf(f[i] * r);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = f[i] * (r * w[i]);
  }
  return pack8(f);
}

// The scaling factor of a row from the sums of squares its warps left in red[].
__device__ __forceinline__ float row_rms_scale(const float* red, int first, int wpr, int K, bool torch_num) {
  float ss = 0.f;
  for (int q = 0; q < wpr; ++q) ss += red[first + q];
  // reference PyTorch RMSNorm: bf16 mean of bf16 squares, bf16 rsqrt, two bf16 products
  // (a one-element bf16 rsqrt on the CPU is 1 / bf16(sqrt(x)) rounded again)
  return torch_num ? torch_rsqrt_bf16(rbf(ss / (float)K), true) : rsqrtf(ss / (float)K + 1e-6f);
}

// A normalised row of at most NV vectors per lane, kept in registers between the sum of
// squares and the scaling; the norm weights were loaded ahead of the op's barrier.
template <int NV>
__device__ __forceinline__ void stage_row_regs(Ctx& c, const uint4* src, uint4* dst, const uint4* pre_w, int K, int nvec,
                                               int v0, int vstep, bool active, bool valid, int red_first, int wpr,
                                               bool gather, int tok, uint4* sum_row) {
  const int kvec = K >> 3;
  const bool torch_num = c.p.numerics == NUM_TORCH;
  float* red = c.red();
  uint4 raw[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int v = v0 + vstep * i;
    raw[i] = (valid && v < kvec && !gather) ? __ldcg(src + v) : make_uint4(0, 0, 0, 0);
  }
  if (gather) {  // (kept apart from the plain loads above: a call between them would serialise them)
#if MK_WITH_XCHG
    if constexpr (NV == 2) {
      // both vectors of a rank in flight together, the ranks one after the other: `world` round trips, not 2 x world
      const KParams& p = c.p;
      const unsigned seq = xchg_cur(c);
      float acc[2][8];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[i][e] = 0.f;
#pragma unroll 1
      for (int r = 0; r < p.world; ++r) {
        uint4 q[2][4];
        const uint4* src4[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int v = min(v0 + vstep * i, kvec - 1);
          src4[i] = reinterpret_cast<const uint4*>(reinterpret_cast<const uint2*>(p.xchg[p.rank]) +
                                                   xchg_word(seq, p.world, p.xchg_tokens, p.xchg_cols, r, tok, v * 8));
#pragma unroll
          for (int k = 0; k < 4; ++k) q[i][k] = (valid && v0 + vstep * i < kvec) ? ld_sys_words(src4[i] + k) : make_uint4(0u, seq, 0u, seq);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if (!(valid && v0 + vstep * i < kvec)) continue;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            if (!xchg_arrived(q[i][k].y, seq) || !xchg_arrived(q[i][k].w, seq)) {
              const uint2* w2 = reinterpret_cast<const uint2*>(src4[i] + k);
              if (xchg_wait_word(c, w2, seq, r) && xchg_wait_word(c, w2 + 1, seq, r)) q[i][k] = ld_sys_words(src4[i] + k);
            }
            acc[i][2 * k] += __uint_as_float(q[i][k].x);
            acc[i][2 * k + 1] += __uint_as_float(q[i][k].z);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int v = v0 + vstep * i;
        if (valid && v < kvec) {
          raw[i] = pack8(acc[i]);
          if (sum_row != nullptr) sum_row[v] = raw[i];  // the reduced row, for a later reader of the tensor itself (a residual)
        }
      }
    } else
#endif
    {
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int v = v0 + vstep * i;
        if (valid && v < kvec) {
          raw[i] = xchg_gather8(c, xchg_cur(c), tok, v * 8);
          if (sum_row != nullptr) sum_row[v] = raw[i];
        }
      }
    }
  }
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) ss = sumsq8(raw[i], torch_num, ss);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if (c.lane == 0) red[c.warp] = ss;
  consumer_sync();
  if (active) {
    const float r = row_rms_scale(red, red_first, wpr, K, torch_num);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = v0 + vstep * i;
      if (v < nvec) dst[x_vec(v)] = scale8(raw[i], pre_w[i], r, torch_num);
    }
  }
  consumer_sync();
}

// `gather`: the rows are not read from `in` but summed over the ranks' slots of the latest exchange.
__device__ __forceinline__ void stage_x(Ctx& c, const void* in, int ld_in, int K, int kp, const void* norm_w, int tok0,
                                     int rows, int T, const uint4* pre_w, bool gather = false, void* sums_out = nullptr) {
  if (!MK_WITH_XCHG) gather = false;  // (compiled out of the single-GPU build)
  uint4* xs = reinterpret_cast<uint4*>(c.smem + c.p.x_off);
  const int pitch = x_pitch(kp);  // uint4 per row
  const int nvec = kp >> 3, kvec = K >> 3;
  const bool torch_num = c.p.numerics == NUM_TORCH;
  const uint4* wv = reinterpret_cast<const uint4*>(norm_w);
  const int wpr = stage_warps_per_row(rows);
  const int tb = c.warp / wpr, part = c.warp % wpr;
  const bool active = tb < rows;
  const bool valid = active && tok0 + tb < T;
  const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(in) + (size_t)(tok0 + tb) * ld_in);
  uint4* dst = xs + tb * pitch;
  float* red = c.red();
  const int v0 = part * 32 + c.lane, vstep = 32 * wpr;
  if (wv != nullptr && pre_w != nullptr && nvec <= 4 * vstep) {
    uint4* sum_row = (gather && sums_out != nullptr && valid) ? reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(sums_out) + (size_t)(tok0 + tb) * ld_in)
                                                              : nullptr;
    if (nvec <= 2 * vstep) stage_row_regs<2>(c, src, dst, pre_w, K, nvec, v0, vstep, active, valid, tb * wpr, wpr, gather, tok0 + tb, sum_row);
    else stage_row_regs<4>(c, src, dst, pre_w, K, nvec, v0, vstep, active, valid, tb * wpr, wpr, gather, tok0 + tb, sum_row);
    return;
  }
  float ss = 0.f;
  if (active) {
    // four loads in flight at a time (a store to shared memory between two loads would
    // order them: the compiler cannot tell the two address spaces apart here)
#pragma unroll 1
    for (int vb = v0; vb < nvec; vb += 4 * vstep) {
      uint4 val[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int v = vb + i * vstep;
        val[i] = (valid && v < kvec && !gather) ? __ldcg(src + v) : make_uint4(0, 0, 0, 0);
      }
      if (gather) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int v = vb + i * vstep;
          if (valid && v < kvec) val[i] = xchg_gather8(c, xchg_cur(c), tok0 + tb, v * 8);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int v = vb + i * vstep;
        if (v < nvec) {
          dst[x_vec(v)] = val[i];
          if (wv != nullptr) ss = sumsq8(val[i], torch_num, ss);
        }
      }
    }
  }
  if (wv != nullptr) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (c.lane == 0) red[c.warp] = ss;
    consumer_sync();
    if (active) {
      const float r = row_rms_scale(red, tb * wpr, wpr, K, torch_num);
#pragma unroll 2
      for (int v = v0; v < kvec; v += vstep)  // a lane re-reads only what it wrote itself
        dst[x_vec(v)] = scale8(dst[x_vec(v)], __ldg(wv + v), r, torch_num);
    }
  }
  consumer_sync();
}

// Staging for a row-owner linear WITHOUT a fused norm (one or two token rows, at most 24 stages
// of 512 k): warp w stages the w-th 64-wide slice of every stage, all in one round of loads and without a CTA-wide sync.  Lane
// l takes the 16-byte chunk (l & 7) of the slices of stages (l >> 3) + 4 i.
// (The same scheme with the norm fused in was 0.36 ms per step SLOWER: its unrolled scaling code
// is several KB that every op would run once, out of a cold instruction cache.)
__device__ __forceinline__ void stage_x_rows(Ctx& c, const void* in, int ld_in, int K, int kp, int tok0, int rows, int T) {
  constexpr int kMaxV = 6;  // 24 stages / 4 per round
  uint4* xs = reinterpret_cast<uint4*>(c.smem + c.p.x_off);
  const int pitch = x_pitch(kp);  // uint4 per row
  const int v0 = ((c.lane >> 3) * kRowsStageK + c.warp * 64 + (c.lane & 7) * 8) >> 3;  // vector of the first round
  constexpr int vstep = 4 * kRowsStageK / 8;                                           // vectors per round
  const int kvec = K >> 3, nvec = kp >> 3;
#pragma unroll 1
  for (int t = 0; t < rows; ++t) {
    const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(in) + (size_t)(tok0 + t) * ld_in);
    const bool live = tok0 + t < T;
    uint4 raw[kMaxV];
#pragma unroll
    for (int i = 0; i < kMaxV; ++i) {
      const int v = v0 + i * vstep;
      raw[i] = (live && v < kvec) ? __ldcg(src + v) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int i = 0; i < kMaxV; ++i) {
      const int v = v0 + i * vstep;
      if (v < nvec) xs[t * pitch + x_vec(v)] = raw[i];
    }
  }
  __syncwarp();
}

// The same two stagings for an input that arrives as tagged words (no barrier stands before the op):
// every lane first issues all its loads, then polls whatever has not arrived.  They are separate
// functions on purpose: folded into the plain ones above they slowed those down by 8 % of a step
// (registers and stack of code that runs once per op).
template <int NV>
__device__ __forceinline__ void stage_ll_regs(Ctx& c, const uint4* ll, uint4* dst, const uint4* pre_w, const uint4* wv, int K,
                                              int nvec, int v0, int vstep, bool active, bool valid, int red_first, int wpr,
                                              unsigned tag) {
  const int kvec = K >> 3;
  const bool torch_num = c.p.numerics == NUM_TORCH;
  float* red = c.red();
  uint4 raw[NV];
  int at[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) at[i] = valid && v0 + vstep * i < kvec ? v0 + vstep * i : -1;
  ll_take(c, ll, at, tag, raw);
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) ss = sumsq8(raw[i], torch_num, ss);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if (c.lane == 0) red[c.warp] = ss;
  consumer_sync();
  if (active) {
    const float r = row_rms_scale(red, red_first, wpr, K, torch_num);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = v0 + vstep * i;
      if (v < nvec) dst[x_vec(v)] = scale8(raw[i], pre_w != nullptr ? pre_w[i] : (v < kvec ? __ldg(wv + v) : make_uint4(0, 0, 0, 0)), r, torch_num);
    }
  }
  consumer_sync();
}
// fused norm; the host only plans it for rows of at most four vectors per lane
__device__ __forceinline__ void stage_x_ll(Ctx& c, const void* ll_in, int ld_in, int K, int kp, const void* norm_w, int tok0,
                                        int rows, int T, const uint4* pre_w, unsigned tag) {
  uint4* xs = reinterpret_cast<uint4*>(c.smem + c.p.x_off);
  const int pitch = x_pitch(kp);
  const int nvec = kp >> 3;
  const int wpr = stage_warps_per_row(rows);
  const int tb = c.warp / wpr, part = c.warp % wpr;
  const bool active = tb < rows;
  const bool valid = active && tok0 + tb < T;
  const uint4* ll = reinterpret_cast<const uint4*>(ll_row(ll_in, ld_in, valid ? tok0 + tb : 0));
  uint4* dst = xs + tb * pitch;
  const int v0 = part * 32 + c.lane, vstep = 32 * wpr;
  const uint4* wv = reinterpret_cast<const uint4*>(norm_w);
  if (nvec <= 2 * vstep) stage_ll_regs<2>(c, ll, dst, pre_w, wv, K, nvec, v0, vstep, active, valid, tb * wpr, wpr, tag);
  else stage_ll_regs<4>(c, ll, dst, pre_w, wv, K, nvec, v0, vstep, active, valid, tb * wpr, wpr, tag);
}
// no norm: every warp stages its own k slices (see stage_x_rows)
__device__ __forceinline__ void stage_rows_ll(Ctx& c, const void* ll_in, int ld_in, int K, int kp, int tok0, int rows, int T, unsigned tag) {
  constexpr int kMaxV = 6;
  uint4* xs = reinterpret_cast<uint4*>(c.smem + c.p.x_off);
  const int pitch = x_pitch(kp);
  const int v0 = ((c.lane >> 3) * kRowsStageK + c.warp * 64 + (c.lane & 7) * 8) >> 3;
  constexpr int vstep = 4 * kRowsStageK / 8;
  const int kvec = K >> 3, nvec = kp >> 3;
#pragma unroll 1
  for (int t = 0; t < rows; ++t) {
    const bool live = tok0 + t < T;
    const uint4* ll = reinterpret_cast<const uint4*>(ll_row(ll_in, ld_in, live ? tok0 + t : 0));
    uint4 raw[kMaxV];
    int at[kMaxV];
#pragma unroll
    for (int i = 0; i < kMaxV; ++i) at[i] = live && v0 + i * vstep < kvec ? v0 + i * vstep : -1;
    ll_take(c, ll, at, tag, raw);
#pragma unroll
    for (int i = 0; i < kMaxV; ++i)
      if (v0 + i * vstep < nvec) xs[t * pitch + x_vec(v0 + i * vstep)] = raw[i];
  }
  __syncwarp();
}

// ------------------------------------------------------------------------------------
// linear layers: pieces shared by the row-owner path (below) and the wide path (mk_wide.cuh)
// ------------------------------------------------------------------------------------
struct ArgBest {
  float v;
  int i;
};
__device__ __forceinline__ ArgBest arg_better(ArgBest a, ArgBest b) {
  // larger value wins; ties go to the lower index
  if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
  return a;
}
__device__ __forceinline__ ArgBest warp_argmax(ArgBest a) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgBest b;
    b.v = __shfl_xor_sync(0xffffffffu, a.v, o);
    b.i = __shfl_xor_sync(0xffffffffu, a.i, o);
    a = arg_better(a, b);
  }
  return a;
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}


// ------------------------------------------------------------------------------------
// Row-owner linear (F_ROWS): for one or two tokens the cross-CTA finish of a k-split costs
// more than the whole weight stream of a small layer, so every CTA takes whole output rows
// instead: a contiguous range of 8-row units, walked in chunks of up to 32 rows over the
// full K.  The token rows are resident in shared memory (stage_x, fused norm included).
//
// A stage holds a chunk's rows for 512 k-elements as eight boxes of 32 rows x 64 k.  Four boxes are the 128 rows of a tcgen05.mma
// whose lane 32 q + r is row r, slice q of the stage (q + 4 for the other four): the k slices of a row lie side by side on the M
// side.  The B operand holds the eight slices of the token row as eight columns (and those of a second token as eight more), so of
// a lane's columns only its own slice's means anything, which costs nothing (a 128 x 16 x 16 product takes as long as a 128 x 64 x
// 16 one) and spares the finish over CTAs.  The issuer (rows_mma_loop) keeps even and odd k steps apart: four accumulators of 16
// columns per chunk, two sets of them in turn, so that the next chunk is multiplied while the warps finish the last.  Warp w takes
// slice w of its lanes' rows from them; the eight partial sums of an output meet in shared memory.  (These are the sums, in the
// order, that mma.sync by the eight warps gave, and the same bits.  With it a stage was in shared memory until the slowest
// warp had multiplied it, a chunk's finish stopped the stream's consumer, and stages could not go to tensor memory.  12 layers of
// 8B width, us per step: one request 1086 -> 1006, two 1146 -> 1042; four layers 1024 wide 127 -> 119; 8 MoE layers 551 -> 552, two
// requests 676 -> 697, whose chunks of two stages are too short to gain from it: now 540 and 679, 582 and 751 before the elected
// producer.)
// ------------------------------------------------------------------------------------
// The token rows of an op (or pass) are staged: the issuer may multiply.
__device__ __forceinline__ void rows_x_ready(const Ctx& c) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the tensor core reads them through the async proxy
  __syncwarp();
  if (c.lane == 0) mbar_arrive(c.xfull_bar(0));
}
// This warp's slice of a chunk's sums -> the sums block: row = lane, `ntok` tokens to columns half, half + 1
__device__ __forceinline__ void rows_take_sums(Ctx& c, int ntok, int half) {
  const int TP = c.p.sums_stride;
  mbar_wait(c, c.acc_full_bar(c.acc_runs & 1), (c.acc_runs >> 1) & 1u, ST_TIMEOUT_FULL);
  __syncwarp();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t acc = c.tmem + (c.acc_runs & 1) * kRowsAccCols + (uint32_t)((c.warp >> 2) * 32 + c.warp) + ((uint32_t)(c.warp & 3) << 21);
  const uint32_t even0 = tmem_ld1(acc), odd0 = tmem_ld1(acc + 16);
  uint32_t even1 = 0u, odd1 = 0u;
  if (ntok > 1) {
    even1 = tmem_ld1(acc + 8);
    odd1 = tmem_ld1(acc + 24);
  }
  tmem_wait_ld();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncwarp();
  if (c.lane == 0) mbar_arrive(c.acc_empty_bar(c.acc_runs & 1));
  c.acc_runs += 1;
  float* d = c.sums() + (c.warp * kChunkRows + c.lane) * TP + half;
  d[0] = __uint_as_float(even0) + __uint_as_float(odd0);
  if (ntok > 1) d[1] = __uint_as_float(even1) + __uint_as_float(odd1);
}
// Tokens one pass of a row-owner linear covers (aux3, fixed by the host from the shared-memory
// budget) and the passes its weight stream makes for T active tokens.
__device__ __forceinline__ int linear_passes(const OpDesc& op, int T) { return (T + op.aux3 - 1) / op.aux3; }
__device__ __forceinline__ void rows_range(const OpDesc& op, int& row0, int& row1, bool& any) {
  const unsigned U = (unsigned)(op.n + kUnitRows - 1) / kUnitRows;
  const unsigned G = min((unsigned)gridDim.x, U);
  any = blockIdx.x < G;
  row0 = any ? (int)tile_begin(blockIdx.x, U, G) * kUnitRows : 0;
  row1 = any ? (int)tile_begin(blockIdx.x + 1, U, G) * kUnitRows : 0;
}
// The CTA's rows are walked in chunks of at most 32 rows, sized as evenly as whole 8-row units
// allow (40 rows are 24 + 16, not 32 + 8: small chunks mean small stages and few bytes in
// flight).  Chunk ci of nch covers rows [rows_chunk_begin(ci), rows_chunk_begin(ci + 1)).
__device__ __forceinline__ int rows_num_chunks(int row0, int row1) { return (row1 - row0 + kChunkRows - 1) / kChunkRows; }
__device__ __forceinline__ int rows_chunk_begin(int row0, int row1, int nch, int ci) {
  return row0 + kUnitRows * (ci * ((row1 - row0) / kUnitRows) / nch);
}
__device__ __forceinline__ void linear_pass_rows(Ctx& c, const OpDesc& op, int tok0, int T, const uint4* pre_w) {
  const KParams& p = c.p;
  const int nks = op.nkt;
  const int kp = nks * kRowsStageK;
  const int ntok = min(op.aux3, T - tok0);
  int row0, row1;
  bool any;
  rows_range(op, row0, row1, any);
  if (!any) return;  // (nor may it poll for tagged words that no output of its own protects from being overwritten)
  MK_STAMP(c, 0);
  if (op.flags & F_LL_IN) {
    if (op.flags & F_NORM_IN) stage_x_ll(c, op.ll_in, op.ld_in, op.k, kp, op.norm_w, tok0, ntok, T, pre_w, ll_tag_of(c, op.ll_in_op));
    else stage_rows_ll(c, op.ll_in, op.ld_in, op.k, kp, tok0, ntok, T, ll_tag_of(c, op.ll_in_op));
  } else if (nks <= 24 && ntok <= 2 && !(op.flags & F_NORM_IN) && !MK_XF(op, F_GATHER_IN)) stage_x_rows(c, op.in, op.ld_in, op.k, kp, tok0, ntok, T);
  else stage_x(c, op.in, op.ld_in, op.k, kp, (op.flags & F_NORM_IN) ? op.norm_w : nullptr, tok0, ntok, T, pre_w,
               MK_XF(op, F_GATHER_IN) != 0);
  rows_x_ready(c);
  MK_STAMP(c, 1);
  const int lane = c.lane;
  const int TP = p.sums_stride;  // token slots of the sums block: [warp][32 rows][TP]
  float* sums = c.sums();
  const bool with_res = (op.flags & F_RESIDUAL) && (!(op.flags & F_RES_RANK0) || p.rank == 0);
  const __nv_bfloat16* res = reinterpret_cast<const __nv_bfloat16*>(op.res);
  __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(op.out);
  // epilogue role of this thread: output (row e & 31, token e >> 5) of the chunk
  const int e_row = c.tid & 31, e_tok = c.tid >> 5;
  ArgBest best;  // F_ARGMAX: lane 0 of warp t keeps the running best of token t over the CTA's rows
  best.v = -INFINITY;
  best.i = 0x7fffffff;
  const int nch = rows_num_chunks(row0, row1);
#pragma unroll 1
  for (int ci = 0; ci < nch; ++ci) {
    const int r0 = rows_chunk_begin(row0, row1, nch, ci);
    const int R = rows_chunk_begin(row0, row1, nch, ci + 1) - r0;
    // the residual of this thread's output is requested a whole chunk ahead of its use
    float res0 = 0.f;
    const bool e_live = e_row < R && e_tok < ntok && r0 + e_row < op.n;
    if (with_res && e_live) {
      if (op.flags & F_LL_RES) res0 = ll_gather1(c, ll_row(op.ll_res, op.ld_res, tok0 + e_tok), r0 + e_row, ll_tag_of(c, op.ll_res_op));
      else res0 = MK_XF(op, F_GATHER_RES) ? xchg_gather1(c, xchg_cur(c), tok0 + e_tok, r0 + e_row)
                                            : __bfloat162float(__ldcg(res + (size_t)(tok0 + e_tok) * op.ld_res + r0 + e_row));
    }
    if (ci == 0) MK_STAMP(c, 2);
    rows_take_sums(c, ntok, 0);
    if (ci == nch - 1) MK_STAMP(c, 3);
    consumer_sync();
    if (op.flags & F_SILU_MUL) {
      // units are [4 gate rows | 4 up rows]: the thread of a gate row also adds up its partner
      const int col = ((r0 + e_row) >> 3) * 4 + (e_row & 3);
      const bool mine = (e_row & 7) < 4 && e_live && col < (op.n >> 1);
      __nv_bfloat16 y = __float2bfloat16_rn(0.f);
      if (mine) {
        float g = 0.f, u = 0.f;
#pragma unroll
        for (int w = 0; w < kNumConsumerWarps; ++w) {
          g += sums[(w * kChunkRows + e_row) * TP + e_tok];
          u += sums[(w * kChunkRows + e_row + 4) * TP + e_tok];
        }
        g = rbf(g);  // the linear output is bf16 before the activation
        u = rbf(u);
        const float sv = rbf(__fdividef(g, 1.0f + __expf(-g)));
        y = __float2bfloat16_rn(sv * u);
        out[(size_t)(tok0 + e_tok) * op.ld_out + col] = y;
      }
      if (op.flags & F_LL_OUT) {  // the pair (col, col + 1) sits in two neighbouring lanes
        const uint32_t lo = (uint32_t)__bfloat16_as_ushort(y);
        const uint32_t hi = __shfl_down_sync(0xffffffffu, lo, 1);
        if (mine && !(e_row & 1))
          st_gpu_word(reinterpret_cast<uint2*>(op.ll_out) + (size_t)(tok0 + e_tok) * (size_t)(op.ld_out >> 1) + (col >> 1), lo | (hi << 16),
                    ll_tag_of(c, c.cur_op));
      }
    } else {
      float v = 0.f;
      if (e_live) {
#pragma unroll
        for (int w = 0; w < kNumConsumerWarps; ++w) v += sums[(w * kChunkRows + e_row) * TP + e_tok];
        if (with_res) v = (p.numerics == NUM_TORCH && !MK_XF(op, F_PUSH)) ? rbf(v) + res0 : v + res0;
        if (MK_XF(op, F_PUSH)) xchg_push1(p, xchg_next(c), tok0 + e_tok, r0 + e_row, v);
        else out[(size_t)(tok0 + e_tok) * op.ld_out + r0 + e_row] = __float2bfloat16_rn(v);
      }
      if (op.flags & F_LL_OUT) {  // rows come in units of 8: the pair (row, row + 1) sits in two neighbouring lanes
        const uint32_t lo = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(v));
        const uint32_t hi = __shfl_down_sync(0xffffffffu, lo, 1);
        if (e_live && !(e_row & 1))
          st_gpu_word(reinterpret_cast<uint2*>(op.ll_out) + (size_t)(tok0 + e_tok) * (size_t)(op.ld_out >> 1) + ((r0 + e_row) >> 1),
                    lo | (hi << 16), ll_tag_of(c, c.cur_op));
      }
      if (op.flags & F_ARGMAX) {
        ArgBest b;
        b.v = e_live ? rbf(v) : -INFINITY;
        b.i = e_live ? r0 + e_row : 0x7fffffff;
        b = warp_argmax(b);
        best = arg_better(best, b);
      }
    }
    if (ci + 1 < nch) consumer_sync();  // the sums block is free again (after the last chunk, the sync that opens the next op or pass does it)
  }
  if ((op.flags & F_ARGMAX) && lane == 0 && e_tok < ntok) {
    op.amax_val[(size_t)(tok0 + e_tok) * op.amax_n + blockIdx.x] = best.v;
    op.amax_idx[(size_t)(tok0 + e_tok) * op.amax_n + blockIdx.x] = best.i;
  }
  MK_STAMP(c, 4);
}

__device__ __forceinline__ void op_linear_rows(Ctx& c, const OpDesc& op, int T) {
  // the norm weights do not depend on other CTAs: fetched ahead of the barrier
  uint4 pre_w[4] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
  const int wpr0 = stage_warps_per_row(min(op.aux3, T));
  const int kvec_pad = op.nkt * (kRowsStageK >> 3);  // padded row, in 16-byte vectors
  const bool pre = (op.flags & F_NORM_IN) && kvec_pad <= 128 * wpr0;
  if (pre) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int v = (c.warp % wpr0) * 32 + c.lane + 32 * wpr0 * i;
      if (v < (op.k >> 3)) pre_w[i] = __ldg(reinterpret_cast<const uint4*>(op.norm_w) + v);
    }
  }
#if MK_WITH_XCHG
  if (op.flags & F_XRED) xchg_reduce_slice(c, op, T);
#endif
  if (op.flags & F_LL_IN) {
    // No barrier, and no look at the abort flag either (a round trip to L2 per op): the polls of the
    // tagged input and the stage waits watch it, and an aborted iteration ends at its closing barrier.
    if (c.pr != nullptr && c.tid == 0) c.pr[1] = globaltimer();
  } else if (op_barrier(c, op)) {
    return;
  }
  c.lin_seq += 1;
  if (c.tid == 0) c.flags()[4] = (int)c.lin_seq;
  const int passes = linear_passes(op, T);
  for (int g = 0; g < passes; ++g) {
    linear_pass_rows(c, op, g * op.aux3, T, (pre && g == 0) ? pre_w : nullptr);
    if (g + 1 < passes) consumer_sync();  // (a pass leaves its last chunk's sums block without a sync of its own)
  }
  if (MK_XF(op, F_PUSH)) c.ar_seq += 1;  // every CTA counts the exchange, with or without rows of its own
}

// ------------------------------------------------------------------------------------
// attention: QK-norm + RoPE + KV append + paged split-KV GQA decode + merge
// ------------------------------------------------------------------------------------
// bf16 reciprocal square root the way the reference PyTorch model's CPU kernels round it:
// `dbl` = scalar loop (sqrt rounded to bf16 before the reciprocal), else vector loop.
__device__ __forceinline__ float torch_rsqrt_bf16(float var, bool dbl) {
  return dbl ? rbf(1.0f / rbf(sqrtf(var))) : rbf(1.0f / sqrtf(var));
}

// The norm weight and the cos/sin rows arrive already loaded (8 bf16 each).  Both halves
// of a warp run this with full-mask shuffles (xor < 16 stays inside a half-warp).
struct F8 {
  float v[8];
};
__device__ __forceinline__ F8 head_norm_rope(F8 xin, uint4 wv, uint4 csv, uint4 snv, int l16, int flags, int numerics,
                                          bool dbl) {
  float* x = xin.v;
  if (flags & F_QK_NORM) {
    float w[8];
    unpack8(wv, w);
    float ss = 0.f;
    if (numerics == NUM_TORCH) {
#pragma unroll
      for (int i = 0; i < 8; ++i) ss += rbf(x[i] * x[i]);
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) ss += x[i] * x[i];
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (numerics == NUM_TORCH) {
      const float r = torch_rsqrt_bf16(rbf(ss / (float)kHeadDim), dbl);
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = rbf(w[i] * rbf(x[i] * r));
    } else {
      const float r = rsqrtf(ss / (float)kHeadDim + 1e-6f);
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = rbf(x[i] * (r * w[i]));
    }
  }
  if (flags & F_ROPE) {
    float cs[8], sn[8];
    unpack8(csv, cs);
    unpack8(snv, sn);
    const float sign = (l16 < 8) ? -1.f : 1.f;  // first half: x*cos - partner*sin
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float other = __shfl_xor_sync(0xffffffffu, x[i], 8);
      if (numerics == NUM_TORCH) x[i] = rbf(rbf(x[i] * cs[i]) + rbf(sign * other * sn[i]));
      else x[i] = rbf(x[i] * cs[i] + sign * other * sn[i]);
    }
  }
  return xin;
}

// Tiles of 16 positions that one CTA of the row-owner path takes alone, see op_attention.  Beyond, the chunks' merge (two round
// trips) costs less than a third round of tiles.  12 layers of 8B width, one request, us per step with 8, 16, 24 and 32:
// 1120, 1112, 1112, 1112 at 200 positions, 1118, 1118, 1135, 1135 at 300, 1124, 1126, 1125, 1163 at 440.
// Outputs that are not the bf16 nearest to a float64 softmax, one and two requests behind 0 to 1200 positions, 1 to 8 q heads per
// kv head, 19.7 million outputs: 0.0286 %; the scalar fp32 form before it 0.0290 %.  Us per layer of 8B width, scalar form and
// this one: behind 100 positions 18.0 and 11.3, 4000 53 and 22, 30000 334 and 44; two requests behind 8000 153 and 30.
constexpr int kAttnSoloTiles = 16;
constexpr int kAttnLensMax = 128;  // requests (the host admits at most 128 batched tokens)

// Merge of a (request, kv head)'s chunks by the CTA that arrived last: only a handful of CTAs per layer ever run it.
// One round of loads: every thread fetches, for its
// output elements, the chunks' values together with their (max, sum) pairs and rescales as it
// goes, eight chunks at a time (more loads in flight per thread measured slower).
__device__ __forceinline__ void attn_merge(Ctx& c, const float* base, __nv_bfloat16* out, int nch, int qpk, int part_stride,
                                        uint2* ll_out, unsigned tag) {
  const int nout = qpk * kHeadDim;
  constexpr int kMergeBatch = 8;
  // a thread merges outputs e and e + 256 side by side: one round of loads for up to eight chunks of both
#pragma unroll 1
  for (int e = c.tid; e < nout; e += 2 * kNumConsumers) {
    const bool two = e + kNumConsumers < nout;
    const int e2 = two ? e + kNumConsumers : e;
    const float* pm = base + nout + (e >> 7);
    const float* pm2 = base + nout + (e2 >> 7);
    float M = -INFINITY, Ls = 0.f, O = 0.f, M2 = -INFINITY, Ls2 = 0.f, O2 = 0.f;
#pragma unroll 1
    for (int c0 = 0; c0 < nch; c0 += kMergeBatch) {
      float v[kMergeBatch], mm[kMergeBatch], ll[kMergeBatch], v2[kMergeBatch], mm2[kMergeBatch], ll2[kMergeBatch];
#pragma unroll
      for (int u = 0; u < kMergeBatch; ++u) {
        const bool ok = c0 + u < nch;
        const size_t off = (size_t)(c0 + u) * part_stride;
        v[u] = ok ? __ldcg(base + off + e) : 0.f;
        mm[u] = ok ? __ldcg(pm + off) : -INFINITY;
        ll[u] = ok ? __ldcg(pm + off + qpk) : 0.f;
        v2[u] = ok ? __ldcg(base + off + e2) : 0.f;
        mm2[u] = ok ? __ldcg(pm2 + off) : -INFINITY;
        ll2[u] = ok ? __ldcg(pm2 + off + qpk) : 0.f;
      }
      float Mb = M, Mb2 = M2;
#pragma unroll
      for (int u = 0; u < kMergeBatch; ++u) {
        Mb = fmaxf(Mb, mm[u]);
        Mb2 = fmaxf(Mb2, mm2[u]);
      }
      const float r = exp2f(M - Mb), r2 = exp2f(M2 - Mb2);  // 0 for the first batch (every chunk holds at least one position)
      O *= r;
      Ls *= r;
      O2 *= r2;
      Ls2 *= r2;
#pragma unroll
      for (int u = 0; u < kMergeBatch; ++u) {
        const float f = exp2f(mm[u] - Mb), f2 = exp2f(mm2[u] - Mb2);
        O = fmaf(f, v[u], O);
        Ls = fmaf(f, ll[u], Ls);
        O2 = fmaf(f2, v2[u], O2);
        Ls2 = fmaf(f2, ll2[u], Ls2);
      }
      M = Mb;
      M2 = Mb2;
    }
    const __nv_bfloat16 y = __float2bfloat16_rn(__fdividef(O, Ls)), y2 = __float2bfloat16_rn(__fdividef(O2, Ls2));
    out[e] = y;
    if (two) out[e2] = y2;
    if (ll_out != nullptr) {  // (whole warps take the same trips: nout is a multiple of 128)
      const uint32_t lo = (uint32_t)__bfloat16_as_ushort(y), lo2 = (uint32_t)__bfloat16_as_ushort(y2);
      const uint32_t hi = __shfl_down_sync(0xffffffffu, lo, 1), hi2 = __shfl_down_sync(0xffffffffu, lo2, 1);
      if (!(e & 1)) {
        st_gpu_word(ll_out + (e >> 1), lo | (hi << 16), tag);
        if (two) st_gpu_word(ll_out + (e2 >> 1), lo2 | (hi2 << 16), tag);
      }
    }
  }
}

// The merge without a counter: every chunk stores its partial (output sums, then max and sum per q head) as
// tagged 8-byte words, and every chunk CTA then merges its own slice of the output elements, polling the
// words of all chunks it needs: no atomic round trip, no last arriver doing all of it, one output per
// thread.  (A CTA stores its own partial before it waits for any other, and the chunks of one pair are
// consecutive tasks, so a wait never depends on a later task of the waiting CTA.)
__device__ __forceinline__ void attn_merge_ll(Ctx& c, const uint2* base, __nv_bfloat16* out, uint2* ll_out, int nch, int ch, int qpk,
                                           int part_stride, unsigned tag) {
  const int nout = qpk * kHeadDim;
  const int S = (((nout + nch - 1) / nch) + 1) & ~1;  // outputs per chunk CTA, even: a bf16 pair never straddles two slices
#pragma unroll 1
  for (int el0 = 0; el0 < S; el0 += kNumConsumers) {  // (one round for up to four q heads per kv head)
    const int el = el0 + c.tid;
    const int e = ch * S + el;
    const bool act = el < S && e < nout;
    float y = 0.f;
    if (act) {
      constexpr int kBatch = 8;
      const uint2* pv = base + e;
      const uint2* pm = base + nout + (e >> 7);
      float M = -INFINITY, Ls = 0.f, O = 0.f;
#pragma unroll 1
      for (int c0 = 0; c0 < nch; c0 += kBatch) {
        uint2 qv[kBatch], qm[kBatch], ql[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
          const unsigned t = c0 + u < nch ? ~tag : tag;
          qv[u] = ql[u] = make_uint2(0u, t);
          qm[u] = make_uint2(0xff800000u, t);  // (-inf)
        }
        PollLimit limit;
        while (true) {
          bool here = true;
#pragma unroll
          for (int u = 0; u < kBatch; ++u) {
            const size_t off = (size_t)(c0 + u) * part_stride;
            if (qv[u].y != tag) qv[u] = ld_gpu_word(pv + off);
            if (qm[u].y != tag) qm[u] = ld_gpu_word(pm + off);
            if (ql[u].y != tag) ql[u] = ld_gpu_word(pm + off + qpk);
          }
#pragma unroll
          for (int u = 0; u < kBatch; ++u) here = here && qv[u].y == tag && qm[u].y == tag && ql[u].y == tag;
          if (here || limit.expired(c, tag, qv[0].y)) break;
        }
        float v[kBatch], mm[kBatch], ll[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
          v[u] = __uint_as_float(qv[u].x);
          mm[u] = __uint_as_float(qm[u].x);
          ll[u] = __uint_as_float(ql[u].x);
        }
        float Mb = M;
#pragma unroll
        for (int u = 0; u < kBatch; ++u) Mb = fmaxf(Mb, mm[u]);
        const float r = exp2f(M - Mb);  // 0 for the first batch (every chunk holds at least one position)
        O *= r;
        Ls *= r;
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
          const float f = exp2f(mm[u] - Mb);
          O = fmaf(f, v[u], O);
          Ls = fmaf(f, ll[u], Ls);
        }
        M = Mb;
      }
      y = __fdividef(O, Ls);
    }
    const __nv_bfloat16 yb = __float2bfloat16_rn(y);
    if (act) out[e] = yb;
    const uint32_t lo = (uint32_t)__bfloat16_as_ushort(yb);
    const uint32_t hi = __shfl_down_sync(0xffffffffu, lo, 1);
    if (act && ll_out != nullptr && !(e & 1)) st_gpu_word(ll_out + (e >> 1), lo | (hi << 16), tag);
  }
}

// Prompt chunks (several tokens of one request in an iteration).  Waits for the op's barrier, then one
// warp per (token, kv head) pair normalises and rotates the token's new K and stores it, with its V, at
// the token's own position in the cache; a second grid barrier makes all of them visible.  Returns true
// when the launch is aborting.  (Both halves of a warp compute the same pair: the shuffles in
// head_norm_rope use the full mask.)
__device__ __forceinline__ bool attn_barrier_then_append(Ctx& c, const OpDesc& op, const int* lens, int T) {
  const KParams& p = c.p;
  const int HKV = op.aux0, qpk = op.aux1 / op.aux0;
  if (op.flags & F_SYNC_BEFORE) {
    grid_wait(c);
    if (c.pr != nullptr && c.tid == 0) c.pr[1] = globaltimer();
    c.dead = c.flags()[3] != 0;
    if (c.dead) return true;
  } else if (op.flags & F_LL_IN) {
    // no barrier stands before this op, but a prompt chunk reads the plain rows of every token: a full one here
    grid_sync(c);
    if (c.pr != nullptr && c.tid == 0) c.pr[1] = globaltimer();
    c.dead = c.flags()[3] != 0;
    if (c.dead) return true;
  } else if (op_barrier(c, op)) {
    return true;
  }
  const int l16 = c.lane & 15;
  const bool dbl_k = op.aux0 < 32;
  const uint4 wk = __ldg(reinterpret_cast<const uint4*>(op.k_norm_w) + l16);
#pragma unroll 1
  for (int pair = blockIdx.x * kNumConsumerWarps + c.warp; pair < T * HKV; pair += gridDim.x * kNumConsumerWarps) {
    const int t = pair / HKV, h = pair % HKV;
    const int L = lens[t];
    if (L <= 0) continue;
    const int pos = min(L - 1, op.aux2 - 1);
    const uint4 cs = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(op.cos) + (size_t)pos * kHeadDim) + l16);
    const uint4 sn = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(op.sin) + (size_t)pos * kHeadDim) + l16);
    const __nv_bfloat16* row = reinterpret_cast<const __nv_bfloat16*>(op.in) + (size_t)t * op.ld_in + (size_t)h * (qpk + 2) * kHeadDim;
    const uint4 vnew = __ldcg(reinterpret_cast<const uint4*>(row + (qpk + 1) * kHeadDim) + l16);
    F8 kf;
    unpack8(__ldcg(reinterpret_cast<const uint4*>(row + qpk * kHeadDim) + l16), kf.v);
    kf = head_norm_rope(kf, wk, cs, sn, l16, op.flags, p.numerics, dbl_k);
    const int pg = __ldcg(p.kv_indices + lens[kAttnLensMax + t] + ((L - 1) >> p.page_shift));
    if (c.lane < 16) {
      const size_t dst = ((((size_t)pg << p.page_shift) + ((L - 1) & (p.page_size - 1))) * HKV + h) * kHeadDim;
      reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(op.k_cache) + dst)[l16] = pack8(kf.v);
      reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(op.v_cache) + dst)[l16] = vnew;
    }
  }
  grid_sync(c);
  c.dead = c.flags()[3] != 0;
  return c.dead;
}

#include "mk_wide.cuh"

// attend_combine for a whole CTA with a slot of shared memory for every warp (16 KB): all of them leave their sums, meet once, and an
// output's thread takes the eight from there, in the order and with the roundings of the two steps that half the slots need.
// Us per step: one request of 12 layers of 8B width 997 -> 989, of four 1024 wide 119.6 -> 117.2, 8 MoE layers 551 -> 545.
template <class Emit>
__device__ __forceinline__ void rows_combine(const Ctx& c, int rows, uint8_t* reg, float2* ml, float m, float l, const float (&oacc)[8][4], Emit emit) {
  constexpr int H = kNumConsumerWarps / 2;
  const int g = c.lane >> 2, j = c.lane & 3;
  if (j == 0) ml[c.warp * 8 + g] = make_float2(m, l);
  float* slot0 = reinterpret_cast<float*>(reg);
#pragma unroll
  for (int rb = 0; rb < 2; ++rb) {
    if (4 * rb >= rows) break;
    if (rb > 0) consumer_sync();  // (the slots are free again)
    if ((j >> 1) == rb) {         // this lane holds rows 2 j and 2 j + 1
      float* own = slot0 + (size_t)c.warp * 4 * kHeadDim + 2 * (j & 1) * kHeadDim + 8 * g;
#pragma unroll
      for (int y = 0; y < 2; ++y)
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
          for (int i = 0; i < 8; i += 4)
            *reinterpret_cast<float4*>(own + y * kHeadDim + 64 * x + i) =
                make_float4(oacc[i][2 * x + y], oacc[i + 1][2 * x + y], oacc[i + 2][2 * x + y], oacc[i + 3][2 * x + y]);
    }
    consumer_sync();
    const int r = 4 * rb + (c.tid >> 5), d = (c.tid & 31) * 4;
    if (c.tid < 4 * 32 && r < rows) {
      float M = -INFINITY;
#pragma unroll
      for (int w = 0; w < kNumConsumerWarps; ++w) M = fmaxf(M, ml[w * 8 + r].x);
      const float Ms = M == -INFINITY ? 0.f : M;
      float L = 0.f;
      float4 O = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int w = 0; w < H; ++w) {
        const float2 v0 = ml[w * 8 + r], v1 = ml[(w + H) * 8 + r];
        L = fmaf(exp2f(v0.x - Ms), v0.y, L);
        L = fmaf(exp2f(v1.x - Ms), v1.y, L);
        const float Mp = fmaxf(v0.x, v1.x), Mps = Mp == -INFINITY ? 0.f : Mp;
        const float f0 = exp2f(v0.x - Mps), f1 = exp2f(v1.x - Mps), f = exp2f(Mp - Ms);
        const float4 a = *reinterpret_cast<const float4*>(slot0 + (size_t)w * 4 * kHeadDim + (c.tid >> 5) * kHeadDim + d);
        const float4 b = *reinterpret_cast<const float4*>(slot0 + (size_t)(w + H) * 4 * kHeadDim + (c.tid >> 5) * kHeadDim + d);
        O.x = fmaf(f, fmaf(f1, b.x, f0 * a.x), O.x);
        O.y = fmaf(f, fmaf(f1, b.y, f0 * a.y), O.y);
        O.z = fmaf(f, fmaf(f1, b.z, f0 * a.z), O.z);
        O.w = fmaf(f, fmaf(f1, b.w, f0 * a.w), O.w);
      }
      emit(rb, r, d, O, M, L);
    }
  }
}

// aux0 = kv heads, aux1 = q heads (q heads per kv head: 1, 2, 4 or 8).  The row-owner path's attention: one or two tokens.
// Latency is all: a task is (token, kv head[, chunk of positions]), done by a whole CTA, whose warps take 16-position tiles in
// turn on the tensor cores (attend_tiles).  The K and V rows of a warp's first tile are requested before the q rows are awaited; q
// heads and the new K are normalised and rotated once per CTA, into shared memory, and the new token's K and V rows are taken
// from there.  (In scalar fp32, a q head per half-warp, a CTA took 16 positions a round at four q heads per kv head: from 17
// positions on the task was split over CTAs and merged across them, 4 us.  12 layers of 8B width, one request, us per step: 1103 ->
// 1088 behind 80 positions, 1199 -> 1132 behind 1000; 8 MoE layers 640 -> 593; 4 layers 1024 wide 134 -> 128.)
__device__ __forceinline__ void op_attention(Ctx& c, const OpDesc& op, int T) {
  const KParams& p = c.p;
  const int G = gridDim.x;
  MK_STAMP(c, 0);
  if (p.debug_flags & 2) {  // measurement aid: the op keeps its barrier and does nothing else
    op_barrier(c, op);
    return;
  }
  // arrive at the op's barrier first: everything up to the wait below is independent of other CTAs
  if (op.flags & F_SYNC_BEFORE) grid_arrive(c);
  const int HKV = op.aux0, qpk = op.aux1 / op.aux0;
  // Per-iteration cache in the scratch region (nothing else touches these bytes): sequence lengths incl. the new token [128],
  // page-table offsets [128], whether some request has several tokens, then the plan.
  int* lens = reinterpret_cast<int*>(c.red() + 64);
  int* multi = lens + 2 * kAttnLensMax;
  int* plan = multi + 1;  // [0] chunk size, [1] chunks of the longest request: the same in every layer of an iteration
  const int key = (c.iter << 8) ^ (op.aux0 * 16 + op.aux1);  // iteration and head geometry
  if (c.attn_iter != key) {
    c.attn_iter = key;
    if (c.tid == 0) *multi = 0;
    consumer_sync();
    // Token t of request r (qo_indptr[r] <= t < qo_indptr[r + 1]) sits at position kv_len(r) - (tokens of r behind
    // it) - 1: its sequence length, itself included, is what the tasks below call L0.
#pragma unroll 1
    for (int r = c.tid; r < p.max_reqs; r += kNumConsumers) {
      const int q0 = __ldcg(p.qo_indptr + r), q1 = min(__ldcg(p.qo_indptr + r + 1), T);
      if (q1 > q0) {
        const int first = __ldcg(p.kv_indptr + r), last = __ldcg(p.kv_indptr + r + 1);
        const int kvlen = (last - first - 1) * p.page_size + __ldcg(p.kv_last_page_len + r);
        for (int t = q0; t < q1; ++t) {
          lens[t] = kvlen - (q1 - 1 - t);
          lens[kAttnLensMax + t] = first;
        }
        if (q1 - q0 > 1) *multi = 1;
      }
    }
    consumer_sync();
    if (c.tid == 0) {
      int tiles = 1;
      for (int t = 0; t < T; ++t) tiles = max(tiles, (lens[t] + 15) >> 4);
      // One CTA per (token, kv head) up to kAttnSoloTiles tiles; beyond, chunks of at least 8 tiles (a tile per warp), as many as one
      // round of CTAs holds.
      int nch = tiles <= kAttnSoloTiles ? 1 : max(1, min(min(G / (T * HKV), (tiles + 7) / 8), p.attn_max_chunks));
      const int tpc = (tiles + nch - 1) / nch;
      plan[0] = tpc * 16;
      plan[1] = (tiles + tpc - 1) / tpc;
    }
    consumer_sync();
  }
  const bool chunked = *multi != 0;
  const int CS = plan[0], nch = plan[1], ntasks = T * HKV * nch;
  const int l16 = c.lane & 15, g = c.lane >> 2, j = c.lane & 3;
  // x region: combine slots [8 warps][4 rows][128] fp32, (max, sum) pairs [8][8], the new token's K and V rows, q rows of pitch 272 bytes
  uint8_t* xr = c.smem + c.p.x_off;
  float2* ml = reinterpret_cast<float2*>(xr + kRowsCombineBytes);
  uint4* sm_k = reinterpret_cast<uint4*>(xr + kRowsCombineBytes + 512);  // [16] K, [16] V
  __nv_bfloat16* sm_q = reinterpret_cast<__nv_bfloat16*>(xr + kRowsCombineBytes + 512 + 512);
  constexpr int kQPitch = 136;
  const bool dbl_q = op.aux1 < 32, dbl_k = op.aux0 < 32;
  const int kw = qpk & 7;  // the warp that prepares the new k (warp 0 when all eight prepare q heads)
  const int part_stride = qpk * (kHeadDim + 2);
  const unsigned tag_in = ll_tag_of(c, op.ll_in_op), tag = ll_tag_of(c, c.cur_op);
  if (chunked) {
    // A prompt chunk: its tokens attend to each other's K/V, which only exist once every token's K has been
    // normalised, rotated and appended.  So this iteration appends first, for all tokens, behind the op's
    // own barrier, and meets at one more grid barrier before any row is read (nothing is fetched early).
    if (attn_barrier_then_append(c, op, lens, T)) return;
  }
  bool first = !chunked;
#pragma unroll 1
  for (int task = blockIdx.x;; task += G) {
    WideTask a;
    a.p0 = a.p1 = a.fresh = a.L0 = 0;
    int ti = c.warp, ntiles = 0, pgn = 0, new_page = 0;
    uint4 kr[2][4], vr[4][2];
    bool live = task < ntasks;
    if (live) {
      a.ch = task % nch;
      a.h = (task / nch) % HKV;
      a.t0 = task / (nch * HKV);
      a.nt = 1;
      a.L0 = lens[a.t0];
      a.kvb = lens[kAttnLensMax + a.t0];
      a.p0 = a.ch * CS;
      a.p1 = min(a.L0, a.p0 + CS);
      a.nch = (a.L0 + CS - 1) / CS;
      a.fresh = chunked ? a.L0 + 16 : a.L0 - 1;  // (a prompt chunk's rows are all in the cache)
      live = a.L0 > 0 && a.p0 < a.L0;
    }
    if (live) {
      ntiles = (a.p1 - a.p0 + 15) >> 4;
      if (ti < ntiles) {
        const int pg = p.page_shift >= 4 ? wide_page(c, a, a.p0 + 16 * ti) : 0;
        wide_load_k(c, op, a, a.p0 + 16 * ti, pg, kr);
        wide_load_v(c, op, a, a.p0 + 16 * ti, pg, vr);
        if (p.page_shift >= 4 && ti + kNumConsumerWarps < ntiles) pgn = wide_page(c, a, a.p0 + 16 * (ti + kNumConsumerWarps));
      }
      if (a.p1 == a.L0) new_page = __ldcg(p.kv_indices + a.kvb + ((a.L0 - 1) >> p.page_shift));
    }
    if (first) {
      // everything above is independent of this layer's QKV rows: fetched ahead of the barrier
      first = false;
      MK_STAMP(c, 1);
      if (op.flags & F_SYNC_BEFORE) {  // op_barrier, with the wait inlined
        grid_wait(c);
        if (c.pr != nullptr && c.tid == 0) c.pr[1] = globaltimer();
        c.dead = c.flags()[3] != 0;
        if (c.dead) return;
      } else if (op.flags & F_LL_IN) {
        // (no look at the abort flag: the polls of the tagged input watch it)
        consumer_sync();
        if (c.pr != nullptr && c.tid == 0) c.pr[1] = globaltimer();
      } else if (op_barrier(c, op)) {
        return;
      }
    }
    if (task >= ntasks) break;
    if (!live) continue;
    const __nv_bfloat16* row = reinterpret_cast<const __nv_bfloat16*>(op.in) + (size_t)a.t0 * op.ld_in + (size_t)a.h * (qpk + 2) * kHeadDim;
    const bool do_q = c.warp < qpk, do_k = c.warp == kw;
    if (do_q || do_k) {
      uint4 vnew, xq = make_uint4(0, 0, 0, 0), xk = make_uint4(0, 0, 0, 0);
      // norm weights and the cos/sin row of the position, beside the rows themselves
      const int pos = min(a.L0 - 1, op.aux2 - 1);  // aux2 = rows of the cos/sin tables
      const uint4 nw = __ldg(reinterpret_cast<const uint4*>(do_q ? op.q_norm_w : op.k_norm_w) + l16);
      const uint4 ncs = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(op.cos) + (size_t)pos * kHeadDim) + l16);
      const uint4 nsn = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(op.sin) + (size_t)pos * kHeadDim) + l16);
      if ((op.flags & F_LL_IN) && !chunked) {  // (a prompt chunk has had its barrier)
        const int at[3] = {do_k ? (qpk + 1) * (kHeadDim / 8) + l16 : -1, do_q ? c.warp * (kHeadDim / 8) + l16 : -1, do_k ? qpk * (kHeadDim / 8) + l16 : -1};
        uint4 got[3];
        ll_take(c, reinterpret_cast<const uint4*>(ll_row(op.ll_in, op.ld_in, a.t0) + ((a.h * (qpk + 2) * kHeadDim) >> 1)), at, tag_in, got);
        __syncwarp();
        vnew = got[0];
        xq = got[1];
        xk = got[2];
      } else {
        vnew = __ldcg(reinterpret_cast<const uint4*>(row + (qpk + 1) * kHeadDim) + l16);
        if (do_q) xq = __ldcg(reinterpret_cast<const uint4*>(row + c.warp * kHeadDim) + l16);
        if (do_k) xk = __ldcg(reinterpret_cast<const uint4*>(row + qpk * kHeadDim) + l16);
      }
      if (do_q) {
        F8 q;
        unpack8(xq, q.v);
        q = head_norm_rope(q, nw, ncs, nsn, l16, op.flags, p.numerics, dbl_q);
        if (c.lane < 16) reinterpret_cast<uint4*>(sm_q + c.warp * kQPitch)[l16] = pack8(q.v);  // exact: the values are bf16 already
      }
      if (do_k) {
        F8 kf;
        unpack8(xk, kf.v);
        kf = head_norm_rope(kf, do_q ? __ldg(reinterpret_cast<const uint4*>(op.k_norm_w) + l16) : nw, ncs, nsn, l16, op.flags, p.numerics, dbl_k);
        const uint4 kn = pack8(kf.v);
        if (c.lane < 16) {
          sm_k[l16] = kn;
          sm_k[16 + l16] = vnew;
          if (a.p1 == a.L0 && !chunked) {  // the last chunk appends the new token's K and V to the cache
            const size_t dst = ((((size_t)new_page << p.page_shift) + ((a.L0 - 1) & (p.page_size - 1))) * HKV + a.h) * kHeadDim;
            reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(op.k_cache) + dst)[l16] = kn;
            reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(op.v_cache) + dst)[l16] = vnew;
          }
        }
      }
    }
    consumer_sync();
    MK_STAMP(c, 2);
    uint4 qf[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) qf[i] = g < qpk ? *reinterpret_cast<const uint4*>(sm_q + g * kQPitch + 32 * i + 8 * j) : make_uint4(0, 0, 0, 0);
    float m, l, oacc[8][4];
    attend_tiles<true>(c, op, a, kNumConsumerWarps, ti, pgn, qf, kr, vr, sm_k, m, l, oacc);
    MK_STAMP(c, 3);
    // a thread ends up with at most one (row, four dims) per batch of four rows: kept until the task is known to be finite
    // (words that others poll cannot be taken back)
    float4 keep[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
    float keep_m[2] = {0.f, 0.f}, keep_l[2] = {1.f, 1.f};
    float chk = 0.f;
    rows_combine(c, qpk, xr, ml, m, l, oacc, [&](int rb, int, int, const float4& O, float M, float L) {
      keep[rb] = O;
      keep_m[rb] = M;
      keep_l[rb] = L;
      chk = fmaf(O.x, 0.f, fmaf(O.y, 0.f, fmaf(O.z, 0.f, fmaf(O.w, 0.f, chk))));
    });
    float* part = p.attn_part + (((size_t)a.t0 * HKV + a.h) * p.attn_max_chunks + a.ch) * part_stride;
    // tagged partials (see attn_merge_ll) when the op's output is tagged and the host gave them room
    const bool ll_part = (op.flags & F_LL_OUT) && p.attn_part_ll != nullptr;
    uint2* partw = p.attn_part_ll + (((size_t)a.t0 * HKV + a.h) * p.attn_max_chunks + a.ch) * part_stride;
    __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(op.out) + (size_t)a.t0 * op.ld_out + (size_t)a.h * qpk * kHeadDim;
    uint2* ll_out = (op.flags & F_LL_OUT) ? reinterpret_cast<uint2*>(op.ll_out) + (size_t)a.t0 * (size_t)(op.ld_out >> 1) + ((a.h * qpk * kHeadDim) >> 1)
                                          : nullptr;
    auto store = [&](int r, int d, const float4& O, float M, float L) {
      if (a.nch == 1) {
        const float inv = __fdividef(1.0f, L);
        const uint2 y = make_uint2(pack2(O.x * inv, O.y * inv), pack2(O.z * inv, O.w * inv));
        if ((op.ld_out & 3) == 0) {
          *reinterpret_cast<uint2*>(out + r * kHeadDim + d) = y;
        } else {  // (rows of any pitch are accepted here)
          unsigned short* dst = reinterpret_cast<unsigned short*>(out) + r * kHeadDim + d;
          dst[0] = (unsigned short)y.x;
          dst[1] = (unsigned short)(y.x >> 16);
          dst[2] = (unsigned short)y.y;
          dst[3] = (unsigned short)(y.y >> 16);
        }
        if (ll_out != nullptr) st_gpu_words(reinterpret_cast<uint4*>(ll_out + ((r * kHeadDim + d) >> 1)), y.x, y.y, tag);
      } else if (ll_part) {
        uint4* dst = reinterpret_cast<uint4*>(partw + r * kHeadDim + d);
        st_gpu_words(dst, __float_as_uint(O.x), __float_as_uint(O.y), tag);
        st_gpu_words(dst + 1, __float_as_uint(O.z), __float_as_uint(O.w), tag);
        if (d == 0) {
          st_gpu_word(partw + qpk * kHeadDim + r, __float_as_uint(M), tag);
          st_gpu_word(partw + qpk * kHeadDim + qpk + r, __float_as_uint(L), tag);
        }
      } else {
        *reinterpret_cast<float2*>(part + r * kHeadDim + d) = make_float2(O.x, O.y);
        *reinterpret_cast<float2*>(part + r * kHeadDim + d + 2) = make_float2(O.z, O.w);
        if (d == 0) {
          part[qpk * kHeadDim + r] = M;
          part[qpk * kHeadDim + qpk + r] = L;
        }
      }
    };
    if (bar_any(2, kNumConsumers, chk != 0.f)) {
      attend_exact(p, op, a, kNumConsumerWarps, sm_q, (size_t)0, kQPitch, store);
    } else if (c.tid < 128) {
#pragma unroll
      for (int rb = 0; rb < 2; ++rb) {
        const int r = 4 * rb + (c.tid >> 5), d = (c.tid & 31) * 4;
        if (r < qpk) store(r, d, keep[rb], keep_m[rb], keep_l[rb]);
      }
    }
    MK_STAMP(c, 4);
    if (a.nch > 1 && ll_part) {
      attn_merge_ll(c, partw - (size_t)a.ch * part_stride, out, ll_out, a.nch, a.ch, qpk, part_stride, tag);
    } else if (a.nch > 1) {
      consumer_sync();  // the CTA's partial is complete; thread 0's release below publishes all of it
      MK_STAMP(c, 5);
      volatile int* fl = c.flags();
      unsigned* cnt = p.attn_count + (size_t)a.t0 * HKV + a.h;
      const float* base = p.attn_part + (((size_t)a.t0 * HKV + a.h) * p.attn_max_chunks) * part_stride;
      if (c.tid == 0) {
        unsigned old;
        asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(cnt) : "memory");
        fl[2] = (old == (unsigned)(a.nch - 1)) ? 1 : 0;
      }
      consumer_sync();
      MK_STAMP(c, 6);
      // The chunk that arrives last merges all of them.  (A fixed merger per kv head, polling the
      // counter, measured slower: the last arriver knows at once that it is the last.)
      if (fl[2] != 0) {
        attn_merge(c, base, out, a.nch, qpk, part_stride, ll_out, tag);
        if (c.tid == 0) *cnt = 0u;
      }
    }
    consumer_sync();
    MK_STAMP(c, 7);
  }
}


// ------------------------------------------------------------------------------------
// small ops
// ------------------------------------------------------------------------------------
// aux0 = embedding rows
__device__ __forceinline__ void op_embed(Ctx& c, const OpDesc& op, int T) {
  const int nseg = (op.n + 2047) / 2048;
  const long long* ids = reinterpret_cast<const long long*>(op.in);
  for (int u = blockIdx.x; u < T * nseg; u += gridDim.x) {
    const int tok = u / nseg, seg = u % nseg;
    long long id = __ldcg(ids + (size_t)tok * op.ld_in);
    if (id < 0 || id >= op.aux0) {
      if (c.tid == 0) raise_abort(c, ST_BAD_TOKEN, tok, (int)id);
      id = 0;
    }
    const int col = seg * 2048 + c.tid * 8;
    if (col < op.n) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(op.w) + (size_t)id * op.ld_res + col));
      *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(op.out) + (size_t)tok * op.ld_out + col) = v;
    }
  }
}

// A row that is too wide for shared memory: read once for its sum of squares (in stage_x's order) and once to be scaled.
__device__ __forceinline__ void rmsnorm_wide_row(Ctx& c, const OpDesc& op, int tok) {
  const bool torch_num = c.p.numerics == NUM_TORCH;
  const int kvec = op.n >> 3;
  const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(op.in) + (size_t)tok * op.ld_in);
  uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(op.out) + (size_t)tok * op.ld_out);
  float* red = c.red();
  float ss = 0.f;
#pragma unroll 4
  for (int v = c.tid; v < kvec; v += kNumConsumers) ss = sumsq8(__ldcg(src + v), torch_num, ss);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if (c.lane == 0) red[c.warp] = ss;
  consumer_sync();
  const float r = row_rms_scale(red, 0, kNumConsumerWarps, op.n, torch_num);
#pragma unroll 4
  for (int v = c.tid; v < kvec; v += kNumConsumers) dst[v] = scale8(__ldcg(src + v), __ldg(reinterpret_cast<const uint4*>(op.w) + v), r, torch_num);
  consumer_sync();
}

__device__ __forceinline__ void op_rmsnorm(Ctx& c, const OpDesc& op, int T) {
  const int kp = ((op.n + 63) / 64) * 64;
  // the norm weights do not depend on other CTAs: a CTA that has a row fetches them ahead of the barrier
  uint4 pre_w[4] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
  const bool pre = (kp >> 3) <= 4 * kNumConsumers;
  if (pre && (int)blockIdx.x < T) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int v = c.tid + kNumConsumers * i;
      if (v < (op.n >> 3)) pre_w[i] = __ldg(reinterpret_cast<const uint4*>(op.w) + v);
    }
  }
  if (op_barrier(c, op)) return;
  for (int tok = blockIdx.x; tok < T; tok += gridDim.x) {
    if (pre && !MK_XF(op, F_GATHER_IN)) {
      // up to 8192 columns: the row stays in registers from the load to the store
      const bool torch_num = c.p.numerics == NUM_TORCH;
      const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(op.in) + (size_t)tok * op.ld_in);
      uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(op.out) + (size_t)tok * op.ld_out);
      const int kvec = op.n >> 3;
      uint4 raw[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) raw[i] = c.tid + kNumConsumers * i < kvec ? __ldcg(src + c.tid + kNumConsumers * i) : make_uint4(0, 0, 0, 0);
      float ss = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) ss = sumsq8(raw[i], torch_num, ss);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      float* red = c.red();
      if (c.lane == 0) red[c.warp] = ss;
      consumer_sync();
      const float r = row_rms_scale(red, 0, kNumConsumerWarps, op.n, torch_num);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (c.tid + kNumConsumers * i < kvec) dst[c.tid + kNumConsumers * i] = scale8(raw[i], pre_w[i], r, torch_num);
      consumer_sync();
      continue;
    }
    if (op.n > kNormStagedCols && !MK_XF(op, F_GATHER_IN)) {
      rmsnorm_wide_row(c, op, tok);
      continue;
    }
    // (the sums are also stored into the gathered tensor's own rows when the host asked for it: aux0)
    if (MK_XF(op, F_GATHER_IN)) stage_x(c, nullptr, op.ld_in, op.n, kp, op.w, tok, 1, tok + 1, pre ? pre_w : nullptr, true,
                                         (op.aux0 && pre) ? const_cast<void*>(op.in) : nullptr);
    else stage_x(c, reinterpret_cast<const __nv_bfloat16*>(op.in) + (size_t)tok * op.ld_in, op.ld_in, op.n, kp, op.w, 0, 1, 1,
                 pre ? pre_w : nullptr);
    const uint4* xs = reinterpret_cast<const uint4*>(c.smem + c.p.x_off);
    uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(op.out) + (size_t)tok * op.ld_out);
    for (int v = c.tid; v < (op.n >> 3); v += kNumConsumers) dst[v] = xs[x_vec(v)];
    consumer_sync();
  }
}

// aux0 = columns per [gate | up] block of the input
__device__ __forceinline__ void op_silu_mul(Ctx& c, const OpDesc& op, int T) {
  const int bk = op.aux0;
  const int nvec = op.n >> 3;
  const __nv_bfloat16* in = reinterpret_cast<const __nv_bfloat16*>(op.in);
  __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(op.out);
  const long long rows = (long long)T * (op.aux1 > 0 ? op.aux1 : 1);  // aux1: rows per token (expert slots of a MoE layer)
  for (long long e = (long long)blockIdx.x * kNumConsumers + c.tid; e < rows * nvec;
       e += (long long)gridDim.x * kNumConsumers) {
    const int tok = (int)(e / nvec), col = (int)(e % nvec) * 8;
    const size_t src = (size_t)tok * op.ld_in + (size_t)(col / bk) * 2 * bk + col % bk;
    float g[8], u[8], r[8];
    unpack8(__ldcg(reinterpret_cast<const uint4*>(in + src)), g);
    unpack8(__ldcg(reinterpret_cast<const uint4*>(in + src + bk)), u);
#pragma unroll
    for (int i = 0; i < 8; ++i) r[i] = rbf(g[i] / (1.0f + expf(-g[i]))) * u[i];
    *reinterpret_cast<uint4*>(out + (size_t)tok * op.ld_out + col) = pack8(r);
  }
}

__device__ __forceinline__ ArgBest block_argmax(Ctx& c, ArgBest b) {
  float* scratch = c.red() + 32;
  b = warp_argmax(b);
  if (c.lane == 0) {
    scratch[c.warp * 2] = b.v;
    scratch[c.warp * 2 + 1] = __int_as_float(b.i);
  }
  consumer_sync();
  ArgBest a;
  a.v = scratch[0];
  a.i = __float_as_int(scratch[1]);
  for (int w = 1; w < kNumConsumerWarps; ++w) {
    ArgBest x;
    x.v = scratch[w * 2];
    x.i = __float_as_int(scratch[w * 2 + 1]);
    a = arg_better(a, x);
  }
  consumer_sync();
  return a;
}

// logits [T][n] -> amax_n partial (value, index) pairs per token
__device__ __forceinline__ void op_argmax_partial(Ctx& c, const OpDesc& op, int T) {
  const int np = op.amax_n;
  const int chunk = (op.n + np - 1) / np;
  const __nv_bfloat16* in = reinterpret_cast<const __nv_bfloat16*>(op.in);
  for (int u = blockIdx.x; u < T * np; u += gridDim.x) {
    const int tok = u / np, ck = u % np;
    const int lo = ck * chunk, hi = min(op.n, lo + chunk);
    ArgBest b;
    b.v = -INFINITY;
    b.i = 0x7fffffff;
    for (int i = lo + c.tid; i < hi; i += kNumConsumers) {
      ArgBest x;
      x.v = __bfloat162float(__ldcg(in + (size_t)tok * op.ld_in + i));
      x.i = i;
      b = arg_better(b, x);
    }
    b = block_argmax(c, b);
    if (c.tid == 0) {
      op.amax_val[(size_t)tok * np + ck] = b.v;
      op.amax_idx[(size_t)tok * np + ck] = b.i;
    }
  }
}

// Partial pairs -> int64 token per row.
// One token's winner, by one thread: under a vocabulary-sharded LM head (F_XRANK) the best of all ranks.
__device__ __forceinline__ void argmax_store(Ctx& c, const OpDesc& op, int tok, ArgBest b) {
#if MK_WITH_XCHG
  if (op.flags & F_XRANK) {  // aux0 = first vocabulary index of this rank's shard
    // every rank tells every rank its best (value, global index) of the token; all pick the same winner
    // (larger value, then lower index: the shards are contiguous, so this is the unsharded rule)
    const KParams& p = c.p;
    const unsigned seq = xchg_next(c);
    if (b.i != 0x7fffffff) b.i += op.aux0;
    const size_t mine = (size_t)p.xchg_amax_word + ((size_t)p.rank * p.xchg_tokens + tok) * 2;
    for (int r = 0; r < p.world; ++r) {
      uint2* w = reinterpret_cast<uint2*>(p.xchg[r]) + mine;
      st_sys_word(w, __float_as_uint(b.v), seq);
      st_sys_word(w + 1, (uint32_t)b.i, seq);
    }
    ArgBest g;
    g.v = -INFINITY;
    g.i = 0x7fffffff;
    for (int r = 0; r < p.world; ++r) {
      const uint2* w = reinterpret_cast<const uint2*>(p.xchg[p.rank]) + (size_t)p.xchg_amax_word + ((size_t)r * p.xchg_tokens + tok) * 2;
      if (!xchg_wait_word(c, w, seq, r) || !xchg_wait_word(c, w + 1, seq, r)) break;
      ArgBest x;
      x.v = __uint_as_float(ld_sys_word(w).x);
      x.i = (int)ld_sys_word(w + 1).x;
      g = arg_better(g, x);
    }
    b = g;
  }
#endif
  reinterpret_cast<long long*>(op.out)[(size_t)tok * op.ld_out] = (b.i == 0x7fffffff) ? -1 : (long long)b.i;
}
// the best of a token's partials i0, i0 + step, ...; five of them in flight
__device__ __forceinline__ ArgBest argmax_scan(const OpDesc& op, int tok, int i0, int step) {
  ArgBest b;
  b.v = -INFINITY;
  b.i = 0x7fffffff;
  const float* val = op.amax_val + (size_t)tok * op.amax_n;
  const int* idx = op.amax_idx + (size_t)tok * op.amax_n;
#pragma unroll 1
  for (int i = i0; i < op.amax_n; i += 5 * step) {
    ArgBest x[5];
#pragma unroll
    for (int u = 0; u < 5; ++u) {
      const bool ok = i + u * step < op.amax_n;
      x[u].v = ok ? __ldcg(val + i + u * step) : -INFINITY;
      x[u].i = ok ? __ldcg(idx + i + u * step) : 0x7fffffff;
    }
#pragma unroll
    for (int u = 0; u < 5; ++u) b = arg_better(b, x[u]);
  }
  return b;
}
// Up to 8 tokens CTA 0 reduces them all, a warp per token: it also runs the bookkeeping that reads the result, so
// nothing has to cross CTAs.  (All warps on one token after the other took 12 us for 8 tokens.)  Larger batches are
// spread over the grid (one token per CTA at a time) and pay one more grid barrier so that CTA 0 sees every token.
__device__ __forceinline__ void op_argmax_reduce(Ctx& c, const OpDesc& op, int T) {
  const bool spread = T > kNumConsumerWarps;
  if (spread) {
    for (int tok = blockIdx.x; tok < T; tok += gridDim.x) {
      const ArgBest b = block_argmax(c, argmax_scan(op, tok, c.tid, kNumConsumers));
      if (c.tid == 0) argmax_store(c, op, tok, b);
    }
  } else if (blockIdx.x == 0) {
    if (c.warp < T) {
      const ArgBest b = warp_argmax(argmax_scan(op, c.warp, c.lane, 32));
      if (c.lane == 0) argmax_store(c, op, c.warp, b);
    }
    consumer_sync();
  }
#if MK_WITH_XCHG
  if (op.flags & F_XRANK) c.ar_seq += 1;
#endif
  if (spread) grid_sync(c);
}


#if MK_WITH_MOE
// ------------------------------------------------------------------------------------
// mixture of experts (Qwen3-MoE decode, one or two batched tokens)
// ------------------------------------------------------------------------------------
// The reference runs routing, the two expert linears, SiLU*up and the weighted sum as tasks of their
// own (tasks/blackwell/topk_softmax_sm100.cuh, moe_linear_sm100.cuh, mul_sum_add_sm100.cuh).  Here, at
// one or two tokens, every (token, expert slot) pair is a GEMV: the expert linears run on the row-owner
// path over a VIRTUAL row space of pairs x rows-per-expert.  A CTA owns a contiguous range of it, walks
// it pair by pair in chunks of at most 32 rows, and the chunk's weight rows are the expert's rows of
// the [experts * rows, K] weight (the TMA row coordinate is expert * rows + row).  The producer can
// only run as far ahead as the routing is known: it waits for the consumers to pass the op's barrier.

// aux0 = top-k, aux1 = experts.  in: router logits [T, experts] bf16; amax_val / amax_idx: the runtime's
// routing tables [T, top-k] (fp32 weight, expert id).  One warp per token: fp32 softmax over the experts,
// k rounds of (largest probability, lowest index), weights renormalised over the k picked
// (transformers' Qwen3MoeTopKRouter with norm_topk_prob; reference task: topk_softmax_sm100.cuh:61-290).
// One token, by one warp: `w_out` / `idx_out` and `w_out2` / `idx_out2` (may be null) receive the k weights and expert
// ids.  `words` not null: the logits arrive as tagged words.  Lane l holds experts l, l + 32, ...: the softmax's sum runs
// over them in that order, however the logits arrive (a word holds two neighbouring experts, so two lanes poll it; polled
// once and handed over by shuffles, the layer's gate/up op took 22.9 instead of 22.0 us).  A round is two warp-wide
// integer reductions (a probability's bits grow with it), not five levels of shuffles of (value, index).
__device__ __forceinline__ void moe_route_token(Ctx& c, const __nv_bfloat16* logits, const uint2* words, unsigned tag, int E, int K, float* w_out,
                                             int* idx_out, float* w_out2, int* idx_out2) {
  float v[8];  // up to 256 experts, 8 per lane
  if (words != nullptr) {
    unsigned long long t0 = 0;
    unsigned spins = 0;
    uint2 q[8];
    while (true) {
      bool here = true;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        q[j] = make_uint2(0u, tag);
        if (c.lane + 32 * j < E) q[j] = ld_gpu_word(words + (c.lane >> 1) + 16 * j);
        here = here && q[j].y == tag;
      }
      if (here) break;
      if (((++spins) & 63u) == 0) {
        if (aborted(c)) break;
        const unsigned long long now = globaltimer();
        if (t0 == 0) {
          t0 = now;
        } else if (now - t0 > 2 * c.p.timeout_ns) {
          raise_abort(c, ST_TIMEOUT_DATA, (int)tag, (int)q[0].y);
          break;
        }
      }
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = (c.lane & 1) ? bf_hi(q[i].x) : bf_lo(q[i].x);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = c.lane + 32 * i < E ? __bfloat162float(__ldcg(logits + c.lane + 32 * i)) : 0.f;
  }
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (c.lane + 32 * i < E) mx = fmaxf(mx, v[i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    v[i] = c.lane + 32 * i < E ? expf(v[i] - mx) : 0.f;
    sum += v[i];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  const float inv = 1.0f / sum;
  uint32_t key[8];  // bits of the probability + 1; 0: not an expert, taken, or not a number
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float pr = v[i] * inv;
    key[i] = (c.lane + 32 * i < E && pr >= 0.f) ? __float_as_uint(pr) + 1u : 0u;
  }
  float picked_sum = 0.f, my_w = 0.f;
  int my_e = 0;
#pragma unroll 1
  for (int k = 0; k < K; ++k) {
    uint32_t best = 0u;
    int bi = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (key[i] > best) {  // (a lane's experts come in ascending order: the first of equals is the lowest)
        best = key[i];
        bi = c.lane + 32 * i;
      }
    const uint32_t m = __reduce_max_sync(0xffffffffu, best);
    const int e = __reduce_min_sync(0xffffffffu, best == m && m != 0u ? bi : 0x7fffffff);
    const float pv = m != 0u ? __uint_as_float(m - 1u) : -INFINITY;
    picked_sum += pv;
    if (c.lane == k) {
      my_w = pv;
      my_e = e;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (c.lane + 32 * i == e) key[i] = 0u;  // taken
  }
  if (c.lane < K) {
    if (w_out != nullptr) w_out[c.lane] = my_w / picked_sum;
    if (idx_out != nullptr) idx_out[c.lane] = my_e;
    if (w_out2 != nullptr) w_out2[c.lane] = my_w / picked_sum;
    if (idx_out2 != nullptr) idx_out2[c.lane] = my_e;
  }
}
__device__ __forceinline__ void op_moe_route(Ctx& c, const OpDesc& op, int T) {
  const int E = op.aux1, K = op.aux0;
  const __nv_bfloat16* in = reinterpret_cast<const __nv_bfloat16*>(op.in);
#pragma unroll 1
  for (int t = blockIdx.x * kNumConsumerWarps + c.warp; t < T; t += gridDim.x * kNumConsumerWarps)
    moe_route_token(c, in + (size_t)t * op.ld_in, nullptr, 0u, E, K, op.amax_val + (size_t)t * K, op.amax_idx + (size_t)t * K, nullptr, nullptr);
}

// The CTA's share of the virtual row space of a MoE linear and its walk: pairs x n rows, contiguous ranges
// of 8-row units per CTA, segments that end at pair boundaries, chunks of at most 32 rows inside a segment.
struct MoeWalk {
  int row0, row1;  // the CTA's virtual rows
  int n;           // rows per expert (= per pair)
  bool any;
};
__device__ __forceinline__ MoeWalk moe_walk(const OpDesc& op, int pairs) {
  MoeWalk w;
  w.n = op.n;
  const unsigned U = (unsigned)pairs * (unsigned)(op.n / kUnitRows);
  const unsigned G = min((unsigned)gridDim.x, U);
  w.any = blockIdx.x < G;
  w.row0 = w.any ? (int)tile_begin(blockIdx.x, U, G) * kUnitRows : 0;
  w.row1 = w.any ? (int)tile_begin(blockIdx.x + 1, U, G) * kUnitRows : 0;
  return w;
}

// This CTA's copy of the routing, behind the staged rows: expert ids [T, top-k], then the weights (at most 64 each).
__device__ __forceinline__ int* moe_route_ids(const Ctx& c) { return reinterpret_cast<int*>(c.smem + c.p.x_off + c.p.x_bytes - 512); }
__device__ __forceinline__ float* moe_route_weights(const Ctx& c) { return reinterpret_cast<float*>(moe_route_ids(c) + 64); }

// `rows` tagged rows of K columns -> rows in shared memory, zero padded, by all consumers: four 8-column
// pieces of a thread in flight, then whatever has not arrived is polled.
__device__ __forceinline__ void stage_ll_pairs(Ctx& c, const uint2* base, int ld, int rows, int K, int kp, unsigned tag) {
  uint4* xs = reinterpret_cast<uint4*>(c.smem + c.p.x_off);
  const int pitch = x_pitch(kp), nvec = kp >> 3, kvec = K >> 3, total = rows * nvec;
#pragma unroll 1
  for (int i0 = c.tid; i0 < total; i0 += 4 * kNumConsumers) {
    uint4 got[4];
    int at[4], dst[4];  // (in 16-byte vectors of eight columns: a row of words is ld / 8 of them)
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u * kNumConsumers, r = i / nvec, v = i - r * nvec;
      dst[u] = i < total ? r * pitch + x_vec(v) : -1;
      at[u] = i < total && v < kvec ? r * (ld >> 3) + v : -1;
    }
    ll_take(c, reinterpret_cast<const uint4*>(base), at, tag, got);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (dst[u] >= 0) xs[dst[u]] = got[u];
  }
  consumer_sync();
}

__device__ __forceinline__ void op_moe_down_combine(Ctx& c, const OpDesc& op, int T);

// aux0 = top-k, aux1 = experts, n = rows per expert, k = K.  w: [experts * n, K] bf16 (tmap_w: the four maps of
// the row-owner path over that 2-D view).  in: [T, K] (one row per token) or, with F_MOE_PAIR_IN, [T * top-k, K];
// out: [T * top-k, n].  amax_idx: the routing table.
// F_SILU_MUL (gate/up): n = 2 * inter, and a chunk of R virtual rows holds R / 2 gate rows and the R / 2 up rows that
// belong to them (tmap_w: maps over [2 * experts, inter, K], one box fetches both halves), so the epilogue also has
// SiLU(gate) * up -> out2 [T * top-k, inter]; the activation layer behind it has nothing left to do.
// F_LL_IN (gate/up): no barrier.  The rows (ll_in) and the router logits (ll_res) arrive as tagged words; the rows are
// staged and normalised while the router linear is still at work.
__device__ __forceinline__ void op_moe_linear(Ctx& c, const OpDesc& op, int T) {
  const KParams& p = c.p;
  const bool ll = (op.flags & F_LL_IN) != 0;
  if (ll) {  // (no look at the abort flag either: the polls and the stage waits watch it)
    if (c.pr != nullptr && c.tid == 0) c.pr[1] = globaltimer();
  } else if (op_barrier(c, op)) {
    return;
  }
  const int topk = op.aux0;
  if (op.flags & F_MOE_COMBINE) {
    c.lin_seq += 1;
    if (c.tid == 0) c.flags()[4] = (int)c.lin_seq;  // the routing is visible: the producer may pick this op's expert rows
    op_moe_down_combine(c, op, T);
    return;
  }
  const int pairs = T * topk;
  const MoeWalk wk = moe_walk(op, pairs);
  const bool work = wk.any && wk.row0 < wk.row1;  // (always, with F_LL_IN: the host sees to it)
  const int nks = op.nkt;
  const int kp = nks * kRowsStageK;
  const bool pair_in = (op.flags & F_MOE_PAIR_IN) != 0, silu = (op.flags & F_SILU_MUL) != 0;
  const int p_first = work ? wk.row0 / wk.n : 0, p_last = work ? (wk.row1 - 1) / wk.n : 0;
  // input rows this CTA needs: those of its pairs (the down projection) or of their tokens
  const int in_first = pair_in ? p_first : p_first / topk;
  const int in_last = pair_in ? p_last : p_last / topk;
  const int nrows = in_last - in_first + 1;  // at most 8 (the host admits MoE graphs for one or two tokens)
  if (ll) {
    // the norm weights do not depend on other CTAs: requested before the rows are awaited
    uint4 pre_w[4];
    const int wpr = stage_warps_per_row(nrows);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int v = (c.warp % wpr) * 32 + c.lane + 32 * wpr * i;
      pre_w[i] = v < (op.k >> 3) ? __ldg(reinterpret_cast<const uint4*>(op.norm_w) + v) : make_uint4(0, 0, 0, 0);
    }
    stage_x_ll(c, op.ll_in, op.ld_in, op.k, kp, op.norm_w, in_first, nrows, T, pre_w, ll_tag_of(c, op.ll_in_op));
  }
  if (op.flags & F_MOE_ROUTE) {
    // The routing folded into this op: warp t of EVERY CTA routes token t from the router logits (one or two
    // tokens) and leaves the expert ids and weights in shared memory, for this CTA's producer and for the down
    // projection; without F_LL_IN CTA 0 also stores the runtime's tables, which the later ops of the layer read
    // behind their barriers.
    const bool table = !ll && blockIdx.x == 0;
    if (c.warp < T)
      moe_route_token(c, reinterpret_cast<const __nv_bfloat16*>(op.res) + (size_t)c.warp * op.ld_res,
                      ll ? ll_row(op.ll_res, op.ld_res, c.warp) : nullptr, ll ? ll_tag_of(c, op.ll_res_op) : 0u, op.aux1, topk,
                      table ? op.amax_val + (size_t)c.warp * topk : nullptr, table ? op.amax_idx + (size_t)c.warp * topk : nullptr,
                      moe_route_weights(c) + c.warp * topk, moe_route_ids(c) + c.warp * topk);
    consumer_sync();
    __threadfence_block();
  }
  c.lin_seq += 1;
  if (c.tid == 0) c.flags()[4] = (int)c.lin_seq;  // the routing is visible: the producer may pick this op's expert rows
  if (!work) return;
  if (!ll)
    stage_x(c, reinterpret_cast<const __nv_bfloat16*>(op.in) + (size_t)in_first * op.ld_in, op.ld_in, op.k, kp,
            (op.flags & F_NORM_IN) ? op.norm_w : nullptr, 0, nrows, nrows, nullptr);
  rows_x_ready(c);
  const int TP = p.sums_stride;
  float* sums = c.sums();
  __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(op.out);
  const int e_row = c.tid & 31;
  int half = 0;
#pragma unroll 1
  for (int pr = p_first; pr <= p_last; ++pr) {
    const int seg0 = max(wk.row0, pr * wk.n), seg1 = min(wk.row1, (pr + 1) * wk.n);
    const int nch = rows_num_chunks(seg0, seg1);
#pragma unroll 1
    for (int ci = 0; ci < nch; ++ci) {
      const int r0 = rows_chunk_begin(seg0, seg1, nch, ci);
      const int R = rows_chunk_begin(seg0, seg1, nch, ci + 1) - r0;
      // Consecutive chunks take turns in the two token slots of the sums block: one CTA-wide sync per chunk.
      half ^= 1;
      rows_take_sums(c, 1, half);
      consumer_sync();
      if (c.warp == 0) {
        float v = 0.f;
        if (e_row < R) {
#pragma unroll
          for (int w = 0; w < kNumConsumerWarps; ++w) v += sums[(w * kChunkRows + e_row) * TP + half];
        }
        const int rp = r0 - pr * wk.n;  // the chunk's first row within the pair
        if (silu) {
          const int h2 = R >> 1, inter = wk.n >> 1;
          const float g = rbf(v), u = rbf(__shfl_sync(0xffffffffu, v, (e_row + h2) & 31));
          const int col = (rp >> 1) + (e_row < h2 ? e_row : e_row - h2);
          if (e_row < R) out[(size_t)pr * op.ld_out + (e_row < h2 ? 0 : inter) + col] = __float2bfloat16_rn(v);
          const __nv_bfloat16 y = __float2bfloat16_rn(rbf(g / (1.0f + expf(-g))) * u);
          const uint32_t lo = (uint32_t)__bfloat16_as_ushort(y), hi = __shfl_down_sync(0xffffffffu, lo, 1);
          if (e_row < h2) {
            reinterpret_cast<__nv_bfloat16*>(op.out2)[(size_t)pr * op.ld_out2 + col] = y;
            if ((op.flags & F_LL_OUT) && !(e_row & 1))  // (columns come in groups of four: the pair sits in two neighbouring lanes)
              st_gpu_word(reinterpret_cast<uint2*>(op.ll_out) + (size_t)pr * (size_t)(op.ld_out2 >> 1) + (col >> 1), lo | (hi << 16),
                        ll_tag_of(c, c.cur_op));
          }
        } else if (e_row < R) {
          out[(size_t)pr * op.ld_out + rp + e_row] = __float2bfloat16_rn(v);
        }
      }
    }
  }
}

// The down projection of the experts with the weighted sum folded in (F_MOE_COMBINE).  A CTA owns a range of the n
// OUTPUT rows for all expert slots of a token: per token it stages the token's top-k input rows, then per chunk of
// rows walks the slots (the weight rows are the slot's expert's rows of that chunk), rounds each slot's sums to bf16
// like the linear's output would be, and adds them up slot by slot exactly as the stand-alone weighted sum does
// (bf16 roundings of the PyTorch model, or fp32 fused multiply-adds), + residual.  The per-slot sums of the warps
// alternate between the two token slots of the sums block, so that one CTA-wide sync per slot is enough.
__device__ __forceinline__ void op_moe_down_combine(Ctx& c, const OpDesc& op, int T) {
  const KParams& p = c.p;
  const int topk = op.aux0;
  int row0, row1;
  bool any;
  rows_range(op, row0, row1, any);
  if (!any || row0 >= row1) return;
  const int nks = op.nkt;
  const int kp = nks * kRowsStageK;
  const int TP = p.sums_stride;  // 2
  float* sums = c.sums();
  const bool torch_num = p.numerics == NUM_TORCH;
  const bool ll = (op.flags & F_LL_IN) != 0;  // the slots' rows as tagged words, the routing from this CTA's shared memory
  const __nv_bfloat16* res = reinterpret_cast<const __nv_bfloat16*>(op.res);
  __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(op.out);
  const int e_row = c.tid & 31;
  const int nch = rows_num_chunks(row0, row1);
#pragma unroll 1
  for (int t = 0; t < T; ++t) {
    if (ll) stage_ll_pairs(c, reinterpret_cast<const uint2*>(op.ll_in) + (size_t)t * topk * (size_t)(op.ld_in >> 1), op.ld_in, topk, op.k, kp, ll_tag_of(c, op.ll_in_op));
    else stage_x(c, reinterpret_cast<const __nv_bfloat16*>(op.in) + (size_t)t * topk * op.ld_in, op.ld_in, op.k, kp, nullptr, 0, topk, topk, nullptr);
    rows_x_ready(c);
#pragma unroll 1
    for (int ci = 0; ci < nch; ++ci) {
      const int r0 = rows_chunk_begin(row0, row1, nch, ci);
      const int R = rows_chunk_begin(row0, row1, nch, ci + 1) - r0;
      float comb = 0.f;  // (threads 0..R-1: the running weighted sum of output row r0 + tid)
      float rr = 0.f;
      if (c.tid < R && res != nullptr)
        rr = (op.flags & F_LL_RES) ? ll_gather1(c, ll_row(op.ll_res, op.ld_res, t), r0 + e_row, ll_tag_of(c, op.ll_res_op))
                                   : __bfloat162float(__ldcg(res + (size_t)t * op.ld_res + r0 + e_row));
#pragma unroll 1
      for (int sl = 0; sl < topk; ++sl) {
        const int half = sl & 1;
        rows_take_sums(c, 1, half);
        consumer_sync();
        if (c.tid < R) {
          float v = 0.f;
#pragma unroll
          for (int w = 0; w < kNumConsumerWarps; ++w) v += sums[(w * kChunkRows + e_row) * TP + half];
          const float f = rbf(v);  // the down projection's output is bf16
          const float wgt = ll ? moe_route_weights(c)[t * topk + sl] : __ldcg(op.amax_val + (size_t)t * topk + sl);
          comb = torch_num ? rbf(comb + rbf(f * wgt)) : fmaf(f, wgt, comb);
        }
      }
      if (c.warp == 0) {
        float v = comb;
        if (res != nullptr) v = (torch_num ? rbf(v) : v) + rr;
        if (e_row < R) out[(size_t)t * op.ld_out + r0 + e_row] = __float2bfloat16_rn(v);
        if (op.flags & F_LL_OUT) {  // rows come in units of 8: the pair (row, row + 1) sits in two neighbouring lanes
          const uint32_t lo = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(v));
          const uint32_t hi = __shfl_down_sync(0xffffffffu, lo, 1);
          if (e_row < R && !(e_row & 1))
            st_gpu_word(reinterpret_cast<uint2*>(op.ll_out) + (size_t)t * (size_t)(op.ld_out >> 1) + ((r0 + e_row) >> 1), lo | (hi << 16),
                      ll_tag_of(c, c.cur_op));
        }
      }
      consumer_sync();  // (the next chunk's or token's first slot writes the half the last slot may still be read from)
    }
  }
}

// aux0 = top-k.  in: [T * top-k, n] bf16, amax_val: routing weights [T, top-k], res: [T, n] (may be null), out: [T, n].
// out[t] = bf16( sum over the token's slots of weight * in[pair] ) + residual  (reference task mul_sum_add_sm100.cuh:17-48;
// the PyTorch model adds the slots up in bf16 and the residual in bf16)
__device__ __forceinline__ void op_moe_combine(Ctx& c, const OpDesc& op, int T) {
  const int topk = op.aux0;
  const int nvec = op.n >> 3;
  const __nv_bfloat16* in = reinterpret_cast<const __nv_bfloat16*>(op.in);
  const __nv_bfloat16* res = reinterpret_cast<const __nv_bfloat16*>(op.res);
  __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(op.out);
  const bool torch_num = c.p.numerics == NUM_TORCH;
#pragma unroll 1
  for (int u = blockIdx.x * kNumConsumers + c.tid; u < T * nvec; u += gridDim.x * kNumConsumers) {
    const int t = u / nvec, v = u % nvec;
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.f;
#pragma unroll 1
    for (int sl = 0; sl < topk; ++sl) {
      const float wgt = __ldcg(op.amax_val + (size_t)t * topk + sl);
      float f[8];
      unpack8(__ldcg(reinterpret_cast<const uint4*>(in + (size_t)(t * topk + sl) * op.ld_in) + v), f);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = torch_num ? rbf(acc[i] + rbf(f[i] * wgt)) : fmaf(f[i], wgt, acc[i]);
    }
    if (res != nullptr) {
      float r[8];
      unpack8(__ldcg(reinterpret_cast<const uint4*>(res + (size_t)t * op.ld_res) + v), r);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = (torch_num ? rbf(acc[i]) : acc[i]) + r[i];
    }
    reinterpret_cast<uint4*>(out + (size_t)t * op.ld_out)[v] = pack8(acc);
  }
}
#endif  // MK_WITH_MOE

// ------------------------------------------------------------------------------------
// stand-alone allreduce layer
// ------------------------------------------------------------------------------------
// aux0 = world size, aux1 = this rank.  in: this rank's partial sums [T, n] bf16, out: the sum over
// ranks [T, n] bf16 (fp32 addition in rank order, one rounding: the reference's reduction task,
// tasks/ampere/reduction.cuh:139-166).  The host lowers an allreduce layer to this op only where it
// cannot fold the exchange into the producing linear's epilogue and the consumers' input staging
// (F_PUSH / F_GATHER_*).  Same exchange words as there: every unit of 8 columns is pushed to all
// ranks and then gathered from this rank's own region by the same thread.
__device__ __forceinline__ void op_allreduce(Ctx& c, const OpDesc& op, int T) {
  const KParams& p = c.p;
  if (op_barrier(c, op)) return;
  const int world = op.aux0;
  const int nvec = op.n >> 3;
  if (world <= 1) {  // a single rank: the sum is the input
#pragma unroll 1
    for (int u = blockIdx.x * kNumConsumers + c.tid; u < T * nvec; u += gridDim.x * kNumConsumers) {
      const int row = u / nvec, v = u % nvec;
      reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(op.out) + (size_t)row * op.ld_out)[v] =
          __ldcg(reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(op.in) + (size_t)row * op.ld_in) + v);
    }
    return;
  }
#if MK_WITH_XCHG
  const unsigned seq = xchg_next(c);
#pragma unroll 1
  for (int u = blockIdx.x * kNumConsumers + c.tid; u < T * nvec; u += gridDim.x * kNumConsumers) {
    const int row = u / nvec, v = u % nvec;
    float f[8];
    unpack8(__ldcg(reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(op.in) + (size_t)row * op.ld_in) + v), f);
    const size_t w = xchg_word(seq, p.world, p.xchg_tokens, p.xchg_cols, p.rank, row, v * 8);
#pragma unroll 1
    for (int r = 0; r < world; ++r) {
      uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<uint2*>(p.xchg[r]) + w);
#pragma unroll
      for (int i = 0; i < 4; ++i) st_sys_words(dst + i, __float_as_uint(f[2 * i]), __float_as_uint(f[2 * i + 1]), seq);
    }
    reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(op.out) + (size_t)row * op.ld_out)[v] = xchg_gather8(c, seq, row, v * 8);
  }
  c.ar_seq += 1;
#endif  // (the host launches the tensor-parallel build of this kernel whenever world > 1)
}

// ------------------------------------------------------------------------------------
// continuous-batching bookkeeping between iterations (the consumers of CTA 0)
// ------------------------------------------------------------------------------------
// Same protocol as the reference's offline mode (persistent_kernel.cuh:380-536): append the sampled tokens, retire finished
// requests and free their pages (`finish`: skipped when there are none to append, alone when a launch bounded by max_iters ends);
// compact the survivors, give each one more token, or a chunk of its prompt as far as the iteration's budget goes, and the pages
// it needs, admit new requests (`prepare`).  Returns the active tokens.
//
// All requests at once, thread i for request i (the host admits at most 128): what used to run on along the list are prefix sums, tokens
// cut off at the budget.  Lists of pages and prompt chunks are copied by warps.  One thread took three dependent round trips
// a request: us between two iterations at 1, 8, 32 and 64 requests 7.9, 14, 42 and 90, now 3, 6, 14 and 11.
struct Sum3 {
  int a, b, c;
};
// Sums over the threads before this one; `all`: over all of them.
__device__ __forceinline__ Sum3 book_sums(Ctx& c, Sum3 v, Sum3& all) {
  int* r = reinterpret_cast<int*>(c.red());  // 8 warps x 3
  const Sum3 own = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int a = __shfl_up_sync(0xffffffffu, v.a, o), b = __shfl_up_sync(0xffffffffu, v.b, o), d = __shfl_up_sync(0xffffffffu, v.c, o);
    if (c.lane >= o) {
      v.a += a;
      v.b += b;
      v.c += d;
    }
  }
  if (c.lane == 31) {
    r[c.warp * 3] = v.a;
    r[c.warp * 3 + 1] = v.b;
    r[c.warp * 3 + 2] = v.c;
  }
  consumer_sync();
  all.a = all.b = all.c = 0;
#pragma unroll
  for (int w = 0; w < kNumConsumerWarps; ++w) {
    if (w == c.warp) {
      v.a += all.a;
      v.b += all.b;
      v.c += all.c;
    }
    all.a += r[w * 3];
    all.b += r[w * 3 + 1];
    all.c += r[w * 3 + 2];
  }
  consumer_sync();
  v.a -= own.a;
  v.b -= own.b;
  v.c -= own.c;
  return v;
}
constexpr int kBookReqs = 128;
static_assert(kBookReqs <= kNumConsumers, "a thread per request");
// What a warp copies of a request: n of a list (of row `row`) from `from` on, to `to`.  In the scratch region behind the sums: one for
// each request, on the row-owner path at most two.
struct BookList {
  int row, from, to, n;
};
static_assert(256 + kBookReqs * sizeof(BookList) <= kWideRedBytes, "the lists fit the scratch region");
__device__ __forceinline__ BookList* book_lists(const Ctx& c) { return reinterpret_cast<BookList*>(c.smem + c.p.red_off + 256); }

// Prompt chunks, but for their first tokens
__device__ __forceinline__ void book_chunks(Ctx& c, bool any, bool mine, int i, int rid, int from, int to, int n) {
  if (!any) return;
  const KParams& p = c.p;
  BookList* list = book_lists(c);
  if (i < p.max_reqs) list[i] = {rid, from, to, mine ? n : 0};
  consumer_sync();
#pragma unroll 1
  for (int r = c.warp; r < p.max_reqs; r += kNumConsumerWarps)
    for (int j = 1 + c.lane; j < list[r].n; j += 32) p.input_tokens[list[r].to + j] = __ldcg(p.tokens + (size_t)list[r].row * p.max_seq_len + list[r].from + j);
  consumer_sync();
}
__device__ __forceinline__ int bookkeep(Ctx& c, bool finish, bool prepare, int* table) {
  const KParams& p = c.p;
  BookList* list = book_lists(c);
  const int R = p.max_reqs, i = c.tid, page = p.page_size;
  const bool slot = i < R;
  int rid = slot ? __ldcg(p.request_ids + i) : -1;
  const int q0 = slot ? __ldcg(p.qo_indptr + i) : 0, q1 = slot ? __ldcg(p.qo_indptr + i + 1) : 0;
  const int k0 = slot ? __ldcg(p.kv_indptr + i) : 0, k1 = slot ? __ldcg(p.kv_indptr + i + 1) : 0;
  const int n_old = __ldcg(p.kv_indptr + R), next = __ldcg(p.sched + 2);
  int head = __ldcg(p.sched), tail = __ldcg(p.sched + 1);
  int st = 0, pl = 0;
  if (rid >= 0) {
    st = __ldcg(p.step + rid);
    pl = __ldcg(p.prompt_lengths + rid);
  }
  long long* row = p.tokens + (size_t)max(rid, 0) * p.max_seq_len;
  int freed = 0;
  if (finish && rid >= 0) {
    const int n = q1 - q0;
    for (int j = max(0, pl - st - 1); j < n; ++j)
      if (st + j + 1 < p.max_seq_len) row[st + j + 1] = __ldcg(p.output_tokens + q0 + j);
    st += n;
    p.step[rid] = st;
    if (st + 1 >= p.max_seq_len || (st >= pl && __ldcg(row + st) == p.eos)) {
      freed = k1 - k0;
      rid = -1;
      p.request_ids[i] = -1;
    }
  }
  // a request still inside its prompt gets a chunk of it (as many tokens as the budget allows), a decoding one its single
  // token; either may get nothing when the iteration's budget is spent
  const bool alive = rid >= 0;
  const int left = pl - st, want = alive ? (left > 0 ? min(left, p.max_tokens_per_req) : 1) : 0;
  Sum3 all;
  const Sum3 at = book_sums(c, {freed, alive ? 1 : 0, want}, all);
  const int nrun = all.b;
  int ntok = min(all.c, p.max_tokens);
  if (all.a > 0) {  // pages that are free again, behind the others
    if (slot) list[i] = {0, k0, tail + at.a, freed};
    consumer_sync();
#pragma unroll 1
    for (int r = c.warp; r < R; r += kNumConsumerWarps)
      for (int j = c.lane; j < list[r].n; j += 32) p.page_queue[(list[r].to + j) % p.max_pages] = __ldcg(p.kv_indices + list[r].from + j);
    tail += all.a;
    consumer_sync();
  }
  if (!prepare) {
    if (c.tid == 0) p.sched[1] = tail;
    return 0;
  }
  const int t0 = min(at.c, p.max_tokens), nnew = min(want, p.max_tokens - t0);
  const int have = alive ? k1 - k0 : 0, pages = alive ? max(have, (st + nnew + page - 1) / page) : 0;
  const Sum3 pg = book_sums(c, {pages, pages - have, nnew > 1 ? 1 : 0}, all);
  if (all.b > tail - head) {
    if (pg.b <= tail - head && pg.b + pages - have > tail - head)  // (the first that gets none)
      raise_abort_at(&p, c.iter, -1, ST_OUT_OF_PAGES, rid, pages);
    if (c.tid == 0) p.sched[1] = tail;  // who has ended stays so, their pages free: another launch may follow
    return 0;
  }
  int npages = all.a;
  if (all.b > 0 || npages != n_old) {  // lists change their places: all of them out of the table first
    int* old_idx = n_old <= p.page_entries ? table : p.page_scratch;
#pragma unroll 1
    for (int j = c.tid; j < n_old; j += kNumConsumers) old_idx[j] = __ldcg(p.kv_indices + j);
    if (slot) list[i] = {0, k0, pg.a, have};
    consumer_sync();
#pragma unroll 1
    for (int r = c.warp; r < R; r += kNumConsumerWarps)
      for (int j = c.lane; j < list[r].n; j += 32) p.kv_indices[list[r].to + j] = old_idx[list[r].from + j];
    for (int j = have; j < pages; ++j) p.kv_indices[pg.a + j] = __ldcg(p.page_queue + (head + pg.b + j - have) % p.max_pages);
    head += all.b;
    consumer_sync();
  }
  if (alive) {
    p.request_ids[at.b] = rid;
    p.qo_indptr[at.b] = t0;
    p.kv_indptr[at.b] = pg.a;
    const int last = (st + nnew) % page;
    p.kv_last_page_len[at.b] = last == 0 ? page : last;
    if (nnew > 0) p.input_tokens[t0] = __ldcg(row + st);
  }
  book_chunks(c, all.c > 0, alive, i, rid, st, t0, nnew);
  // new requests: as many of the next ones as there are places, tokens of the budget and pages for
  int nreq = nrun;
  if (nreq < R && ntok < p.max_tokens && next < p.total_requests) {
    const int r = next + i;
    const bool may = i < R - nreq && r < p.total_requests;
    const int w = may ? max(1, min(__ldcg(p.prompt_lengths + r), p.max_tokens_per_req)) : 0;
    const Sum3 s = book_sums(c, {w, 0, 0}, all);
    const int q = ntok + s.a, n = may && q < p.max_tokens ? min(w, p.max_tokens - q) : 0, pgs = (n + page - 1) / page;
    const Sum3 u = book_sums(c, {pgs, 0, 0}, all);
    const bool ok = n > 0 && u.a + pgs <= tail - head;  // (where one has to wait for pages, the later ones do too: the sums grow)
    if (ok) {
      p.request_ids[nreq + i] = r;
      p.qo_indptr[nreq + i] = q;
      p.kv_indptr[nreq + i] = npages + u.a;
      const int last = n % page;
      p.kv_last_page_len[nreq + i] = last == 0 ? page : last;
      for (int j = 0; j < pgs; ++j) p.kv_indices[npages + u.a + j] = __ldcg(p.page_queue + (head + u.a + j) % p.max_pages);
      p.input_tokens[q] = __ldcg(p.tokens + (size_t)r * p.max_seq_len);
    }
    book_sums(c, {ok ? 1 : 0, ok ? n : 0, ok ? pgs : 0}, all);  // (the totals)
    book_chunks(c, all.b > all.a, ok, i, r, 0, q, n);
    nreq += all.a;
    ntok += all.b;
    npages += all.c;
    head += all.c;
  }
  if (slot && i >= nreq) p.request_ids[i] = -1;
  if (i <= R && i >= nreq) {
    p.qo_indptr[i] = ntok;
    p.kv_indptr[i] = npages;
  }
  if (c.tid == 0) {
    p.sched[0] = head;
    p.sched[1] = tail;
    p.sched[2] = next + nreq - nrun;
  }
  return ntok;
}

// ------------------------------------------------------------------------------------
// the TMA producer
// ------------------------------------------------------------------------------------
// Position in this CTA's weight-tile sequence: the linear ops in program order, each
// with the CTA's contiguous tile range.
struct TileCursor {
  int oi;
  unsigned tile, t1;
  int blk, kt, nkt;
  const void* tmap;
  bool valid;
};

// Open the CTA's range of linear op `oi`; false if the op is not linear or gives this CTA nothing.
__device__ __forceinline__ bool cursor_open(const KParams& p, TileCursor& tc, int oi) {
  const OpDesc& op = p.ops[oi];
  if (op.type != OP_LINEAR) return false;
  const unsigned total = (unsigned)op.nblk * (unsigned)op.nkt;
  const int G = wide_ctas((int)gridDim.x, op.nblk, op.nkt);
  if ((int)blockIdx.x >= G) return false;
  tc.oi = oi;
  tc.tile = tile_begin(blockIdx.x, total, G);
  tc.t1 = tile_begin(blockIdx.x + 1, total, G);
  tc.nkt = op.nkt;
  tc.blk = (int)(tc.tile / (unsigned)op.nkt);
  tc.kt = (int)(tc.tile - (unsigned)tc.blk * (unsigned)op.nkt);
  tc.tmap = op.tmap_w;
  return tc.tile < tc.t1;
}

// Step the look-ahead cursor one tile, wrapping from the last linear op to the first
// (the next iteration streams the same weights).
__device__ __forceinline__ void cursor_advance_wrap(const KParams& p, TileCursor& tc) {
  tc.tile += 1;
  if (++tc.kt == tc.nkt) {
    tc.kt = 0;
    tc.blk += 1;
  }
  if (tc.tile < tc.t1) return;
  int oi = tc.oi;
  for (int n = 0; n < p.num_ops; ++n) {
    oi = (oi + 1 == p.num_ops) ? 0 : oi + 1;
    if (cursor_open(p, tc, oi)) return;
  }
  tc.valid = false;
}

// Position in this CTA's sequence of row-owner stages (op, chunk, k stage), used by the L2
// look-ahead of the producer; wraps from the last linear op to the first.
struct RowsCursor {
  int oi, row0, row1, nch, ci, ks, nks;
  bool valid;
};
__device__ __forceinline__ bool rows_cursor_open(const KParams& p, RowsCursor& rc, int oi) {
  const OpDesc& op = p.ops[oi];
  if (op.type != OP_LINEAR || !(op.flags & F_ROWS)) return false;
  int row0, row1;
  bool any;
  rows_range(op, row0, row1, any);
  if (!any || row0 >= row1) return false;
  rc.oi = oi;
  rc.row0 = row0;
  rc.row1 = row1;
  rc.nch = rows_num_chunks(row0, row1);
  rc.ci = 0;
  rc.ks = 0;
  rc.nks = op.nkt;
  return true;
}
__device__ __forceinline__ void rows_cursor_next(const KParams& p, RowsCursor& rc) {
  if (++rc.ks < rc.nks) return;
  rc.ks = 0;
  if (++rc.ci < rc.nch) return;
  int oi = rc.oi;
  for (int n = 0; n < p.num_ops; ++n) {
    oi = (oi + 1 == p.num_ops) ? 0 : oi + 1;
    if (rows_cursor_open(p, rc, oi)) return;
  }
  rc.valid = false;
}
// L2 look-ahead of the row-owner weight stream, run by the 32 lanes of the (otherwise idle)
// activation-producer warp: the stages the ring will load next are requested into L2 line by
// line with plain prefetch instructions, so that HBM keeps streaming while the consumers sit
// in a barrier or stage their inputs, and the ring refills from L2 when they come back.
__device__ __forceinline__ void rows_prefetch_loop(Ctx& c) {
  const KParams& p = c.p;
  if (p.prefetch_tiles <= 0) return;
  const unsigned W = (unsigned)p.prefetch_tiles;
  volatile int* fl = c.flags();
  RowsCursor rc;
  rc.valid = false;
  for (int oi = 0; oi < p.num_ops && !rc.valid; ++oi) rc.valid = rows_cursor_open(p, rc, oi);
  unsigned pos = 0;  // the cursor's index in this CTA's stage sequence
  while (rc.valid) {
    if (fl[0] < 0) break;  // the consumers have left
    const unsigned issued = (unsigned)fl[1];
    if (pos >= issued + W) {
      __nanosleep(200);
      continue;
    }
    if (pos >= issued) {
      const OpDesc& op = p.ops[rc.oi];
      const int r0 = rows_chunk_begin(rc.row0, rc.row1, rc.nch, rc.ci);
      const int R = rows_chunk_begin(rc.row0, rc.row1, rc.nch, rc.ci + 1) - r0;
      const unsigned char* w = reinterpret_cast<const unsigned char*>(op.w);
      for (int idx = c.lane; idx < R * 8; idx += 32) {
        const int row = r0 + (idx >> 3), kk = rc.ks * kRowsStageK + (idx & 7) * 64;
        if (row < op.n && kk < op.k) {
          const unsigned char* a = w + ((size_t)row * op.ld_out2 + kk) * 2;
          asm volatile("prefetch.global.L2 [%0];" ::"l"(a));
        }
      }
    }
    rows_cursor_next(p, rc);
    ++pos;
  }
}

template <int PATH>
__device__ __forceinline__ void producer_loop(Ctx& c) {
  const KParams& p = c.p;
  const int S = p.num_stages;
  volatile int* fl = c.flags();
  unsigned issued = 0;
  int s = 0;
  uint32_t empty_parity = 1;  // a fresh barrier passes a wait on the "previous" phase
#if MK_WITH_MOE
  unsigned lin_seq = 0;       // linear and MoE-linear ops seen so far in this launch (the consumers count the same way)
#endif
  const uint32_t bar_full0 = c.full_bar(0), bar_empty0 = c.empty_bar(0);
  // look-ahead: tiles beyond the shared-memory ring are requested into L2 so that HBM
  // keeps streaming while the consumers sit in barriers, staging and epilogues
  TileCursor pc;
  pc.valid = false;
  int ahead = 0;
  if (PATH == PATH_WIDE && p.prefetch_tiles > 0)
    for (int oi = 0; oi < p.num_ops && !pc.valid; ++oi) pc.valid = cursor_open(p, pc, oi);
  // Weights are read once per step: their lines are marked evict-first on the way through L2, so
  // that what the look-ahead has fetched (and the KV cache) is not pushed out by bytes already used.
  uint64_t pol_stream;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol_stream));
  for (int iter = 1;; ++iter) {
    // wait for the consumers to publish this iteration's token count (or the end)
    int go;
    {
      unsigned long long t0 = 0;
      int spins = 0;
      while (true) {
        go = fl[0];
        if (go < 0 || (go >> 8) >= iter) break;
        __nanosleep(40);
        if (((++spins) & 255) == 0) {
          if (aborted(c)) { go = -1; break; }
          const unsigned long long now = globaltimer();
          if (t0 == 0) t0 = now;
          if (now - t0 > 4 * c.p.timeout_ns) {
            raise_abort(c, ST_TIMEOUT_GO, iter, go);
            go = -1;
            break;
          }
        }
      }
    }
    if (go < 0) break;
    const int T = go & 255;
    bool dead = false;
    for (int oi = 0; oi < p.num_ops && !dead; ++oi) {
      const OpDesc& rop = p.ops[oi];
      if constexpr (PATH == PATH_ROWS) {
#if MK_WITH_MOE
        if (rop.type == OP_MOE_LINEAR) {
          // the expert of a pair is only known once the consumers have routed the tokens (or passed the op's barrier);
          // a down projection without a barrier takes the experts of the gate/up linear before it: no wait
          lin_seq += 1;
          const bool routed = (rop.flags & F_MOE_ROUTE) != 0 || (rop.flags & (F_MOE_COMBINE | F_LL_IN)) == (F_MOE_COMBINE | F_LL_IN);
          const volatile int* route = moe_route_ids(c);
          if (!((rop.flags & F_MOE_COMBINE) && routed)) {
            unsigned long long t0 = 0;
            int spins = 0;
            while ((unsigned)fl[4] < lin_seq) {
              if (fl[0] < 0) { dead = true; break; }
              __nanosleep(40);
              if (((++spins) & 1023) == 0) {
                if (aborted(c)) { dead = true; break; }
                const unsigned long long now = globaltimer();
                if (t0 == 0) t0 = now;
                if (now - t0 > 4 * c.p.timeout_ns) { dead = true; break; }
              }
            }
          }
          if (dead) break;
          __threadfence();
          const int topk = rop.aux0;
          if (rop.flags & F_MOE_COMBINE) {
            // output rows owned for all slots: token, chunk of rows, slot, k stage (the consumers' order)
            int row0, row1;
            bool any;
            rows_range(rop, row0, row1, any);
            if (!any || row0 >= row1) continue;
            const int nch = rows_num_chunks(row0, row1);
            for (int t = 0; t < T && !dead; ++t)
              for (int ci = 0; ci < nch && !dead; ++ci) {
                const int r0 = rows_chunk_begin(row0, row1, nch, ci);
                const int R = rows_chunk_begin(row0, row1, nch, ci + 1) - r0;
                const void* tmap = reinterpret_cast<const unsigned char*>(rop.tmap_w) + ((R >> 3) - 1) * 128;
                const uint32_t box_bytes = (uint32_t)R * 128u;
                for (int sl = 0; sl < topk && !dead; ++sl) {
                  const int wrow = (routed ? route[t * topk + sl] : __ldcg(rop.amax_idx + t * topk + sl)) * rop.n + r0;
                  for (int ks = 0; ks < rop.nkt; ++ks) {
                    if (!mbar_wait(c, bar_empty0 + 8 * s, empty_parity, ST_TIMEOUT_EMPTY)) {
                      dead = true;
                      break;
                    }
                    const uint32_t full = bar_full0 + 8 * s;
                    const uint32_t dst = c.smem_addr + (uint32_t)s * (uint32_t)p.stage_bytes;
                    mbar_arrive_expect_tx(full, 8u * box_bytes);
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                      tma_load_2d_hint(dst + (uint32_t)(j * kRowsBoxBytes), tmap, full, ks * kRowsStageK + j * kBoxK, wrow, pol_stream);
                    issued += 1;
                    fl[1] = (int)issued;
                    if (++s == S) {
                      s = 0;
                      empty_parity ^= 1u;
                    }
                  }
                }
              }
            continue;
          }
          const MoeWalk wk = moe_walk(rop, T * topk);
          if (!wk.any || wk.row0 >= wk.row1) continue;
          const int p_first = wk.row0 / wk.n, p_last = (wk.row1 - 1) / wk.n;
          for (int pr = p_first; pr <= p_last && !dead; ++pr) {
            const int expert = routed ? route[pr] : __ldcg(rop.amax_idx + pr);
            const bool silu = (rop.flags & F_SILU_MUL) != 0;
            const int seg0 = max(wk.row0, pr * wk.n), seg1 = min(wk.row1, (pr + 1) * wk.n);
            const int nch = rows_num_chunks(seg0, seg1);
            for (int ci = 0; ci < nch && !dead; ++ci) {
              const int r0 = rows_chunk_begin(seg0, seg1, nch, ci);
              const int R = rows_chunk_begin(seg0, seg1, nch, ci + 1) - r0;
              const void* tmap = reinterpret_cast<const unsigned char*>(rop.tmap_w) + ((R >> 3) - 1) * 128;
              const uint32_t box_bytes = (uint32_t)R * 128u;
              const int wrow = expert * wk.n + (r0 - pr * wk.n);  // the chunk's first row in the [experts * n, K] weight
              for (int ks = 0; ks < rop.nkt; ++ks) {
                if (!mbar_wait(c, bar_empty0 + 8 * s, empty_parity, ST_TIMEOUT_EMPTY)) {
                  dead = true;
                  break;
                }
                const uint32_t full = bar_full0 + 8 * s;
                const uint32_t dst = c.smem_addr + (uint32_t)s * (uint32_t)p.stage_bytes;
                mbar_arrive_expect_tx(full, 8u * box_bytes);
#pragma unroll
                for (int j = 0; j < 8; ++j)
                  if (silu) tma_load_3d_hint(dst + (uint32_t)(j * kRowsBoxBytes), tmap, full, ks * kRowsStageK + j * kBoxK, (r0 - pr * wk.n) >> 1, 2 * expert, pol_stream);
                  else tma_load_2d_hint(dst + (uint32_t)(j * kRowsBoxBytes), tmap, full, ks * kRowsStageK + j * kBoxK, wrow, pol_stream);
                issued += 1;
                fl[1] = (int)issued;
                if (++s == S) {
                  s = 0;
                  empty_parity ^= 1u;
                }
              }
            }
          }
          continue;
        }
        if (rop.type == OP_LINEAR) lin_seq += 1;
#endif
        if (rop.type != OP_LINEAR) continue;
        // row-owner op: per chunk of up to 32 owned rows, the full K in 512-wide stages of
        // eight boxes; the tensor map for a chunk of R rows is the (R / 8)-th of the op's four
        int row0, row1;
        bool any;
        rows_range(rop, row0, row1, any);
        if (!any) continue;
        const int passes = linear_passes(rop, T);
        const int nch = rows_num_chunks(row0, row1);
        for (int g = 0; g < passes && !dead; ++g)
          for (int ci = 0; ci < nch && !dead; ++ci) {
            const int r0 = rows_chunk_begin(row0, row1, nch, ci);
            const int R = rows_chunk_begin(row0, row1, nch, ci + 1) - r0;
            const void* tmap = reinterpret_cast<const unsigned char*>(rop.tmap_w) + ((R >> 3) - 1) * 128;
            const uint32_t box_bytes = (uint32_t)R * 128u;
            for (int ks = 0; ks < rop.nkt; ++ks) {
              if (!mbar_wait(c, bar_empty0 + 8 * s, empty_parity, ST_TIMEOUT_EMPTY)) {
                dead = true;
                break;
              }
              const uint32_t full = bar_full0 + 8 * s;
              const uint32_t dst = c.smem_addr + (uint32_t)s * (uint32_t)p.stage_bytes;
              mbar_arrive_expect_tx(full, 8u * box_bytes);
#pragma unroll
              for (int j = 0; j < 8; ++j)
                tma_load_2d_hint(dst + (uint32_t)(j * kRowsBoxBytes), tmap, full, ks * kRowsStageK + j * kBoxK, r0, pol_stream);
              issued += 1;
              fl[1] = (int)issued;
              if (++s == S) {
                s = 0;
                empty_parity ^= 1u;
              }
            }
          }
        continue;
      } else {
      TileCursor lc;
      if (!cursor_open(p, lc, oi)) continue;
      for (; lc.tile < lc.t1; ++lc.tile) {
        if (pc.valid) {
          while (ahead < p.prefetch_tiles) {
            tma_prefetch_2d(pc.tmap, pc.kt * kTileK, pc.blk * kTileRows);
            tma_prefetch_2d(pc.tmap, pc.kt * kTileK + kBoxK, pc.blk * kTileRows);
            cursor_advance_wrap(p, pc);
            ++ahead;
          }
          --ahead;
        }
        if (!mbar_wait(c, bar_empty0 + 8 * s, empty_parity, ST_TIMEOUT_EMPTY)) {
          dead = true;
          break;
        }
        const uint32_t full = bar_full0 + 8 * s;
        const uint32_t dst = c.smem_addr + (uint32_t)s * (uint32_t)kStageBytes;
        mbar_arrive_expect_tx(full, kStageBytes);
        tma_load_2d_hint(dst, lc.tmap, full, lc.kt * kTileK, lc.blk * kTileRows, pol_stream);
        tma_load_2d_hint(dst + kSubBytes, lc.tmap, full, lc.kt * kTileK + kBoxK, lc.blk * kTileRows, pol_stream);
        issued += 1;
        fl[1] = (int)issued;
        if (++s == S) {
          s = 0;
          empty_parity ^= 1u;
        }
        if (++lc.kt == lc.nkt) {
          lc.kt = 0;
          lc.blk += 1;
        }
      }
      }  // wide path
    }
    if (dead || p.mode == MODE_ONEPASS) break;
  }
  fl[1] = (int)issued;
}

#if MK_NC == 0
// ------------------------------------------------------------------------------------
// the MMA issuer of the row-owner path (one elected lane of warp 10)
// ------------------------------------------------------------------------------------
// Walks the chunks in the consumers' order; see linear_pass_rows for the operands and WeightRing for what happens while the token
// rows are not there.
__device__ __forceinline__ void rows_mma_loop(Ctx& c) {
  const KParams& p = c.p;
  volatile int* fl = c.flags();
  WeightRing ring(c, kRowsSlots, c.tmem + 2 * kRowsAccCols);
  // instruction descriptor: D = f32, A = B = bf16, both K-major, N = 16, M = 128
  const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((16u >> 3) << 17) | ((128u >> 4) << 24);
  unsigned runs = 0;  // chunks started
  uint32_t x_parity = 0;
  const uint32_t x0 = c.smem_addr + p.x_off;
  const bool arith = !(p.debug_flags & 1);
  bool dead = false;
  // what a chunk needs besides its token rows: its accumulators and its first tile
  auto open_chunk = [&] { return ring.wait(c.acc_empty_bar(runs & 1), ((runs >> 1) & 1u) ^ 1u) && ring.wait_tile(); };
  // one (open) chunk: the token row (or two, `second` bytes apart) at x
  auto chunk = [&](uint32_t x, uint32_t second, int nks) {
    const uint32_t d0 = c.tmem + (runs & 1u) * kRowsAccCols;
    uint64_t bd = umma_smem_desc(x, second);
#pragma unroll 1
    for (int ks = 0; ks < nks; ++ks) {
      if (ks > 0 && !ring.wait_tile()) return false;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t more = ks > 0 ? 1u : 0u;
      if (ring.held == 0) {
        const uint64_t ad = umma_smem_desc(ring.stage());
        if (arith)
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int k16 = 0; k16 < 4; ++k16)
              umma_bf16(d0 + 32 * h + 16 * (k16 & 1), ad + (uint64_t)(h * (kSubBytes >> 4) + 2 * k16), bd + (uint64_t)(2 * k16), idesc, k16 < 2 ? more : 1u);
        if (ks + 1 == nks) umma_commit(c.acc_full_bar(runs & 1));
        ring.free_stage();
      } else {
        const uint32_t at = ring.slot();
        if (arith)
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int k16 = 0; k16 < 4; ++k16)
              umma_bf16_ta(d0 + 32 * h + 16 * (k16 & 1), at + 32 * h + 8 * k16, bd + (uint64_t)(2 * k16), idesc, k16 < 2 ? more : 1u);
        if (ks + 1 == nks) umma_commit(c.acc_full_bar(runs & 1));
        ring.free_slot();
      }
      bd += 1024 >> 4;
    }
    ++runs;
    return true;
  };
  for (int iter = 1; !dead; ++iter) {
    int go;
    if (!wait_go(c, fl, iter, go)) break;
    const int T = go & 255;
    for (int oi = 0; oi < p.num_ops && !dead; ++oi) {
      const OpDesc& op = p.ops[oi];
      // Short ops wait for this thread: all of the op's words that are used behind a wait are read ahead of it (a wait may have changed
      // memory, so the compiler would read them from there again, 0.4 us between the staged rows and the first product), and the
      // accumulators are handed over before the stage is.  Linears in a row (barrier each) of 512 x 512 4.7 and 4.2 us, 2048 x 2048
      // 5.3 and 4.9; us per step of four layers 1024 wide 117.9 and 115.3, six 512 wide 150.7 and 146.6.
      const int type = op.type, nks = op.nkt, topk = op.aux0, per_pass = op.aux3;
      const uint32_t row_bytes = (uint32_t)nks * 1024u;
      // groups of chunks on the same staged rows; chunks of a group (in a MoE linear: of each of its pairs, on the pair's row or its
      // token's); the down projection goes chunk by chunk, slot by slot
      int groups, chunks = 0, first = 0, last = 0;
#if MK_WITH_MOE
      MoeWalk wk;
      const bool pairs = type == OP_MOE_LINEAR && !(op.flags & F_MOE_COMBINE), slots = type == OP_MOE_LINEAR && !pairs, pair_in = (op.flags & F_MOE_PAIR_IN) != 0;
      if (pairs) {
        wk = moe_walk(op, T * topk);
        if (!wk.any || wk.row0 >= wk.row1) continue;
        groups = 1;
        first = wk.row0 / wk.n;
        last = (wk.row1 - 1) / wk.n;
      } else
#else
      constexpr bool slots = false;
#endif
      {
        if (type != OP_LINEAR && !slots) continue;
        int row0, row1;
        bool any;
        rows_range(op, row0, row1, any);
        if (!any) continue;
        chunks = rows_num_chunks(row0, row1) * (slots ? topk : 1);
        groups = slots ? T : linear_passes(op, T);
      }
      for (int g = 0; g < groups && !dead; ++g) {
        // (of one token the columns of a second hold whatever lies behind the stage's slices)
        const uint32_t second = type == OP_LINEAR && min(per_pass, T - g * per_pass) > 1 ? row_bytes : 1024u;
        // (ahead of the token rows, which come last: no look at the first chunk's accumulators and tile behind them)
        bool open = ring.held > 0 && mbar_test_wait(c.acc_empty_bar(runs & 1), ((runs >> 1) & 1u) ^ 1u);
        dead = !ring.wait(c.xfull_bar(0), x_parity, ring.S - 1);
        x_parity ^= 1u;
        for (int pr = first; pr <= last && !dead; ++pr) {
          uint32_t x = x0;
#if MK_WITH_MOE
          if (pairs) {
            chunks = rows_num_chunks(max(wk.row0, pr * wk.n), min(wk.row1, (pr + 1) * wk.n));
            x += (uint32_t)(pair_in ? pr - first : pr / topk - first / topk) * row_bytes;
          }
#endif
          for (int i = 0; i < chunks && !dead; ++i) {
            dead = !(open || open_chunk()) || !chunk(slots ? x + (uint32_t)(i % topk) * row_bytes : x, second, nks);
            open = false;
          }
        }
      }
    }
    if (p.mode == MODE_ONEPASS) break;
  }
  // nothing of this thread may be in flight when the tensor memory is given back
  umma_commit(c.done_bar());
  mbar_wait(c, c.done_bar(), 0u, ST_TIMEOUT_FULL);
  fl[5] = (int)ring.taken;
}
#endif

// Arrivals that complete a stage's activation boxes: the 32 lanes of the norm warp where an instance has one (a box that needs no
// norm is arrived at 32 times by its producer), else the producer's.
constexpr uint32_t kBoxArrivals = MK_NC != 0 && 2 * MK_NC <= kNormBoxRows ? 32 : 1;

// The activation producer of the wide path (warp 9, one lane).  It walks the same tile sequence
// as the weight producer and loads the input boxes of every tile into a ring of their own, but only after the
// consumers have passed the op's barrier: unlike weights, activations are the previous op's output.
__device__ __forceinline__ void xproducer_loop(Ctx& c) {
  const KParams& p = c.p;
  const int S = p.num_stages;
  volatile int* fl = c.flags();
  int s = 0;
  uint32_t empty_parity = 1;
  unsigned lin_seq = 0;
  // per stage: parity of its next use, whether its latest box is a plain one; raw boxes (for the norm warp) issued and
  // parity of the next one
  unsigned xuse = 0, last_plain = 0, issued_raw = 0, raw_phase = 0;
  const uint32_t bar_x0 = c.xfull_bar(0), bar_raw0 = c.xraw_bar(0), bar_empty0 = c.xempty_bar(0);
  const uint32_t x_sub = (uint32_t)p.x_rows * 128u;
  for (int iter = 1;; ++iter) {
    int go;
    if (!wait_go(c, fl, iter, go)) break;
    bool dead = false;
    for (int oi = 0; oi < p.num_ops && !dead; ++oi) {
      const OpDesc& op = p.ops[oi];
      if (op.type != OP_LINEAR) continue;
      lin_seq += 1;
      TileCursor lc;
      if (!cursor_open(p, lc, oi)) continue;
      const bool raw = (op.flags & F_NORM_IN) != 0;
      const void* tmap = op.tmap_x;
      asm volatile("prefetch.tensormap [%0];" ::"l"(tmap) : "memory");
      if (!wait_lin(c, fl, 4, lin_seq)) {  // the consumers have passed this op's barrier
        dead = true;
        break;
      }
      asm volatile("fence.proxy.async;" ::: "memory");  // the rows were written with plain stores, TMA reads them
      for (; lc.tile < lc.t1; ++lc.tile) {
        if (!mbar_wait(c, bar_empty0 + 8 * s, empty_parity, ST_TIMEOUT_EMPTY)) {
          dead = true;
          break;
        }
        const uint32_t full = (raw ? bar_raw0 : bar_x0) + 8 * s;
        const uint32_t dst = c.xbox(s);
        mbar_arrive_expect_tx(full, 2 * x_sub);
        if (kBoxArrivals > 1 && !raw) mbar_arrive_n(full, kBoxArrivals - 1);
        tma_load_2d(dst, tmap, full, lc.kt * kTileK, 0);
        tma_load_2d(dst + x_sub, tmap, full, lc.kt * kTileK + kBoxK, 0);
        xuse ^= 1u << s;
        if (raw) {
          issued_raw |= 1u << s;
          raw_phase ^= 1u << s;
          last_plain &= ~(1u << s);
        } else {
          last_plain |= 1u << s;
        }
        if (++s == S) { s = 0; empty_parity ^= 1u; }
        if (++lc.kt == lc.nkt) { lc.kt = 0; lc.blk += 1; }
      }
    }
    if (dead || p.mode == MODE_ONEPASS) break;
  }
  // no copy of this thread may still be in flight when the CTA exits
  for (int i = 0; i < S; ++i) {
    if (issued_raw & (1u << i)) mbar_wait(c, bar_raw0 + 8 * i, ((raw_phase >> i) & 1u) ^ 1u, ST_TIMEOUT_FULL);
    if (last_plain & (1u << i)) mbar_wait(c, bar_x0 + 8 * i, ((xuse >> i) & 1u) ^ 1u, ST_TIMEOUT_FULL);
  }
}

// ------------------------------------------------------------------------------------
// the kernel
// ------------------------------------------------------------------------------------
template <int PATH, int NC>
__global__ void __launch_bounds__(kNumThreads, 1) megakernel(const __grid_constant__ KParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // The parameters are read from shared memory: behind a reference they are generic loads, and the L1 left beside the
  // ring (28 KB when this was measured; 92 KB since the wide path keeps to the 164 KB carve-out) does not hold them from op
  // to op.  Measured, 12 layers of 8B width: 1.765 -> 1.720 ms
  // at 8 requests, 2.364 -> 2.321 at 64; one request 0.3207 -> 0.3166 ms on a small model, no change at 8B width.
  __shared__ __align__(16) uint32_t skp[sizeof(KParams) / 4];
  for (int i = threadIdx.x; i < (int)(sizeof(KParams) / 4); i += blockDim.x) skp[i] = reinterpret_cast<const uint32_t*>(&p)[i];
  __syncthreads();
  Ctx c(*reinterpret_cast<const KParams*>(skp));
  // 128-byte-swizzled TMA stages need a 1024-byte-aligned base; the host budgets the slack
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t pad = (1024u - (raw_addr & 1023u)) & 1023u;
  c.smem = smem_raw + pad;
  c.smem_addr = raw_addr + pad;
  c.epoch = p.bar_epoch0;
#if MK_HIER_BARRIER
  c.nbar = 0;
  c.cl_size = p.cluster > 1 ? (uint32_t)p.cluster : 1u;
  c.cl_rank = 0;
  if (c.cl_size > 1) asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(c.cl_rank));
#endif
  c.arrived = false;
  c.attn_iter = -1;
  c.tmem = 0u;
  c.acc_runs = 0;
  c.tid = threadIdx.x;
  c.lane = threadIdx.x & 31;
  c.warp = threadIdx.x >> 5;
  c.iter = 0;
  c.cur_op = -1;
  c.dbg = nullptr;
  c.pr = nullptr;
  c.dead = false;
  c.ar_seq = 0;
  c.lin_seq = 0;
  volatile int* fl = c.flags();
  if (threadIdx.x == 0) {
    for (int s = 0; s < kMaxStages; ++s) {
      mbar_init(c.full_bar(s), 1);
      mbar_init(c.empty_bar(s), 1);  // the commit behind what read the stage
      mbar_init(c.xfull_bar(s), PATH == PATH_WIDE ? kBoxArrivals : kNumConsumerWarps);
      mbar_init(c.xempty_bar(s), 1);
      mbar_init(c.xraw_bar(s), 1);
      mbar_init(c.tfree_bar(s), 1);
    }
    mbar_init(c.done_bar(), 1);
    for (int b = 0; b < 2; ++b) {
      mbar_init(c.acc_full_bar(b), 1);
      mbar_init(c.acc_empty_bar(b), kNumConsumerWarps);
    }
#if MK_HIER_BARRIER
    mbar_init(c.cl_arrive_bar(), c.cl_size);
    mbar_init(c.cl_open_bar(), 1);
#endif
    fl[0] = 0;
    fl[1] = 0;
    fl[2] = 0;
    fl[3] = 0;
    fl[4] = 0;
    fl[5] = 0;
    fl[6] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
#if MK_HIER_BARRIER
  if (c.cl_size > 1) {  // no CTA may arrive on a peer's mbarrier before it is initialised
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
#endif
  // All of the tensor memory (the CTA has its SM to itself), allocated once by warp 0 and freed by it when the CTA leaves: two
  // sets of fp32 accumulators, then slots of the weight ring.
  if (c.warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(c.tmem_slot()), "n"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  c.tmem = *reinterpret_cast<volatile uint32_t*>(c.smem + p.bar_off + kFlagsOff + 72);

  if (c.warp >= kNumConsumerWarps) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(service_regs(NC)));
    if (c.warp == kNumConsumerWarps) {
      // (one elected lane: the compiler then issues TMA and tcgen05 instructions from uniform registers, without moving their operands
      // there one by one.  8 MoE layers, one request 582 -> 551 us per step, two 751 -> 676; one request of 12 dense layers of 8B
      // width 1073 and 1081, and the wide instances spill)
      if (MK_WITH_MOE ? elect_one() : c.lane == 0) producer_loop<PATH>(c);
    } else if (c.warp == kNumConsumerWarps + 1) {
      if constexpr (PATH == PATH_ROWS) {
        rows_prefetch_loop(c);
      } else {
        if (c.lane == 0) xproducer_loop(c);
      }
    } else if (c.warp == kNumConsumerWarps + 2) {
#if MK_NC == 0
      if (elect_one()) rows_mma_loop(c);
#else
      if (elect_one()) mma_loop(c);
#endif
    } else {
      if constexpr (PATH == PATH_WIDE && 2 * NC <= kNormBoxRows) norm_loop(c);
    }
    __syncwarp();
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(consumer_regs(NC)));
    for (int iter = 1;; ++iter) {
      c.iter = iter;
      c.cur_op = -1;
      int T;
      unsigned long long* prof = p.prof;
      if (prof && c.tid == 0) prof[((size_t)p.num_ops * gridDim.x + blockIdx.x) * 4 + 0] = globaltimer();
      if (p.mode == MODE_OFFLINE) {
        if (blockIdx.x == 0) {
          const int prepared = __ldcg(p.sched + 5), appended = __ldcg(p.sched + 4);
          const int git = __ldcg(p.sched + 7) + iter;  // this iteration's number within the call (sched[7]: of earlier kernels)
          int n = 0;
          bool hand_over = false;
          if (!bar_any(1, kNumConsumers, c.tid == 0 && aborted(c))) {  // (all threads take thread 0's view)
            if (iter == 1 && prepared > 0) {
              n = prepared;  // by the kernel that handed this iteration over
            } else {
              // sched[4] != 0: the last iteration's outputs have not been appended yet
              const bool prepare = p.max_iters == 0 || git <= p.max_iters;
              // (the page table goes through the weight ring: no stage is under way between two iterations)
              if (appended != 0 || prepare) n = bookkeep(c, appended != 0, prepare, reinterpret_cast<int*>(c.smem));
              asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // TMA writes there next
              if (c.tid == 0) p.sched[4] = n > 0 ? 1 : 0;
            }
            // not an iteration for this program: leave it prepared and let the host launch the other one
            hand_over = n > 0 && (n < p.tok_lo || n > p.tok_hi);
            if (c.tid == 0) {
              p.sched[5] = hand_over ? n : 0;
              if (hand_over) p.sched[7] = git - 1;
            }
          }
          if (c.tid == 0) {
            if (!hand_over && git - 1 < p.max_step_times) {
              p.step_times[2 * (git - 1)] = globaltimer();
              p.step_times[2 * (git - 1) + 1] = (unsigned long long)n;
            }
            p.sched[3] = git - 1;
            p.ctrl[0] = hand_over ? -2 : (n > 0 ? n : -1);
            __threadfence();
          }
        }
        grid_sync(c);
        T = __ldcg(p.ctrl);
      } else {
        T = (iter == 1) ? __ldcg(p.qo_indptr + p.max_reqs) : -1;
        if (T == 0) T = -1;
      }
      if (aborted(c)) T = -1;
      // the whole CTA must agree: take thread 0's view
      if (c.tid == 0) fl[3] = T;
      consumer_sync();
      T = fl[3];
      consumer_sync();
      if (prof && c.tid == 0) prof[((size_t)p.num_ops * gridDim.x + blockIdx.x) * 4 + 2] = globaltimer();
      if (T <= 0) break;
      if (T > 255) T = 255;
      if (c.tid == 0) fl[0] = (iter << 8) | T;
      if constexpr (PATH == PATH_WIDE) {
        if (p.has_attn) wide_fill_tokens(c, T);
      }

      // The op descriptors are read from a two-slot copy in shared memory: the next op's
      // descriptor is fetched asynchronously while the current op runs, so that no op starts
      // with a round trip to L2 for its own parameters.
      constexpr int kDescVecs = (int)(sizeof(OpDesc) / 16);
      OpDesc* sdesc = reinterpret_cast<OpDesc*>(c.smem + p.desc_off);
      if (c.tid < kDescVecs)
        reinterpret_cast<uint4*>(&sdesc[0])[c.tid] = __ldg(reinterpret_cast<const uint4*>(&p.ops[0]) + c.tid);
      for (int oi = 0; oi < p.num_ops; ++oi) {
        if (c.tid < kDescVecs) asm volatile("cp.async.wait_all;" ::: "memory");
        consumer_sync();
        const OpDesc& op = sdesc[oi & 1];
        if (oi + 1 < p.num_ops && c.tid < kDescVecs) {
          const uint32_t dst = smem_u32(&sdesc[(oi + 1) & 1]) + 16 * c.tid;
          const void* src = reinterpret_cast<const uint4*>(&p.ops[oi + 1]) + c.tid;
          asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
          asm volatile("cp.async.commit_group;" ::: "memory");
        }
        c.cur_op = oi;
        c.opaque();
        unsigned long long* pr = prof ? prof + ((size_t)oi * gridDim.x + blockIdx.x) * 4 : nullptr;
        c.dbg = (prof && oi == p.trace_op) ? prof + ((size_t)(p.num_ops + 1) * gridDim.x) * 4 + (size_t)blockIdx.x * 16 : nullptr;
        if (pr && c.tid == 0) pr[0] = globaltimer();
        c.pr = pr;
        c.dead = false;
        if ((op.flags & F_CTA0_ONLY) && blockIdx.x != 0) {
          if (op_barrier(c, op)) break;
          if (pr && c.tid == 0) pr[2] = pr[1];
          continue;
        }
        switch (op.type) {
          case OP_EMBED: if (!op_barrier(c, op)) op_embed(c, op, T); break;
          case OP_RMSNORM: op_rmsnorm(c, op, T); break;
          case OP_LINEAR:
            if constexpr (PATH == PATH_WIDE) op_linear_wide<NC>(c, op, T);
            else op_linear_rows(c, op, T);
            break;
          case OP_ATTN:
            if constexpr (PATH == PATH_WIDE) op_attention_wide(c, op, T);
            else op_attention(c, op, T);
            break;
          case OP_SILU_MUL:
#if MK_WITH_MOE
            if (op.flags & F_FOLDED) break;  // the expert linear before it has done it
#endif
            if (!op_barrier(c, op)) op_silu_mul(c, op, T);
            break;
          case OP_ARGMAX_PARTIAL: if (!op_barrier(c, op)) op_argmax_partial(c, op, T); break;
          case OP_ARGMAX_REDUCE: if (!op_barrier(c, op)) op_argmax_reduce(c, op, T); break;
          case OP_ALLREDUCE: op_allreduce(c, op, T); break;
#if MK_WITH_MOE
          case OP_MOE_ROUTE: if (!op_barrier(c, op)) op_moe_route(c, op, T); break;
          case OP_MOE_LINEAR: op_moe_linear(c, op, T); break;
          case OP_MOE_COMBINE: if (!op_barrier(c, op)) op_moe_combine(c, op, T); break;
#endif
          default: op_barrier(c, op); break;
        }
        if (pr && c.tid == 0) pr[2] = globaltimer();
        if (c.dead) break;
      }
      if (p.mode == MODE_ONEPASS) break;
      if (aborted(c)) {
        // fall through to the next iteration's uniform abort check
      }
    }
    // the producer may be waiting for the next iteration
    consumer_sync();
    if (c.tid == 0) {
      fl[0] = -1;
      // exchanges executed by this launch: the host advances its running sequence base by it
      if (blockIdx.x == 0) p.sched[6] = (int)c.ar_seq;
    }
  }
  __syncthreads();
  // no CTA may exit with a bulk copy still writing its shared memory
  if (threadIdx.x == 0) {
    const unsigned issued = (unsigned)fl[1];
    for (unsigned i = (unsigned)fl[5]; i < issued; ++i)
      mbar_wait(c, c.full_bar(i % p.num_stages), (i / p.num_stages) & 1, ST_TIMEOUT_FULL);
  }
  __syncthreads();
  if (c.warp == 0) {
    // (the tcgen05 issuer has waited for everything it had in flight)
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(c.tmem), "n"(kTmemCols) : "memory");
  }
#if MK_HIER_BARRIER
  if (c.cl_size > 1) {  // a peer may still be storing into this CTA's shared memory
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
#endif
}

}  // namespace MK_VARIANT
}  // namespace mk

#define MK_CAT3_(a, b, c) a##b##_##c
#define MK_CAT3(a, b, c) MK_CAT3_(a, b, c)
extern "C" const void* MK_CAT3(mk_instance_, MK_VARIANT, MK_NC)() {
  return (const void*)mk::MK_VARIANT::megakernel<MK_NC == 0 ? mk::PATH_ROWS : mk::PATH_WIDE, MK_NC>;
}
