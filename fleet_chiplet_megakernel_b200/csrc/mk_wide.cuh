// The wide path of the megakernel: iterations of 3 to 128 tokens (batches, prompt chunks).
//
// Linears are stream-K tiles on the 5th-generation tensor cores.  Five roles per CTA work side by side:
//   warp 8   weight producer      TMA boxes of 128 rows x 64 k into the ring (producer_loop)
//   warp 9   activation producer  the matching boxes of x_rows token rows x 64 k, in a ring of their own (xproducer_loop)
//   warp 10  MMA issuer           tcgen05.mma over a tile's boxes, accumulators in tensor memory, where it also sets weights
//                                 aside that have to wait for their activations (mma_loop)
//   warp 11  norm warp            RMSNorm of the activation boxes, up to 32 token rows (norm_loop)
//   warps 0-7                     finish: accumulators -> split-k exchange -> epilogue (linear_wide)
// The accumulators are double-buffered, so the MMAs of the next row block run while the finishing warps
// are still busy with the last one.
//
// Included by mk_kernel.cu inside its namespace.

// ------------------------------------------------------------------------------------
// tcgen05
// ------------------------------------------------------------------------------------
// NC (8, 16 or 32) accumulator columns of this warp's 32 lanes; the caller waits with tmem_wait_ld
template <int NC>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[NC]) {
  if constexpr (NC == 8) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
  } else if constexpr (NC == 16) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
  } else {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
  }
}

// This CTA's range of a stream-K linear's tiles (row block major, k minor); false: nothing for it.
__device__ __forceinline__ bool wide_range(const KParams& p, const OpDesc& op, unsigned& total, int& G, unsigned& t0, unsigned& t1) {
  total = (unsigned)op.nblk * (unsigned)op.nkt;
  G = wide_ctas((int)gridDim.x, op.nblk, op.nkt);  // (the rest idle)
  if ((int)blockIdx.x >= G) return false;
  t0 = tile_begin(blockIdx.x, total, G);
  t1 = tile_begin(blockIdx.x + 1, total, G);
  return t0 < t1;
}

// ------------------------------------------------------------------------------------
// token table of the iteration, in the scratch region behind the reduction words
// ------------------------------------------------------------------------------------
// pos[t]: position of token t in its sequence; slot[t]: cache row (page * page size + offset) of that position;
// kvb[t]: first entry of its request in the page table; grp[g]: query groups of the attention (first token |
// tokens << 8 | their count in plan[]).
constexpr int kWideTab = 128;  // the host admits at most 128 batched tokens
struct WideTab {
  int pos[kWideTab], slot[kWideTab], kvb[kWideTab], req[kWideTab], grp[kWideTab];
  int fresh[kWideTab];  // first position of the token's request whose K/V row is written in this iteration
  int plan[8];
  int scan[8];
  // of the linear op at hand: what its input norm multiplies a token's row with (fp32, or a pair of bf16), even tokens first
  alignas(16) uint32_t scale[kNormBoxRows];
};
static_assert(256 + sizeof(WideTab) <= kWideRedBytes, "the token table fits the scratch region");
__device__ __forceinline__ WideTab& wide_tab(const Ctx& c) { return *reinterpret_cast<WideTab*>(c.smem + c.p.red_off + 256); }

// Filled once per iteration, by all consumers.  Token t of request r (qo_indptr[r] <= t < qo_indptr[r + 1]) sits at
// position kv_len(r) - (tokens of r behind it) - 1.
__device__ __forceinline__ void wide_fill_tokens(Ctx& c, int T) {
  const KParams& p = c.p;
  WideTab& tab = wide_tab(c);
  T = min(T, kWideTab);
#pragma unroll 1
  for (int r = c.tid; r < p.max_reqs; r += kNumConsumers) {
    const int q0 = __ldcg(p.qo_indptr + r), q1 = min(__ldcg(p.qo_indptr + r + 1), T);
    if (q1 > q0) {
      const int first = __ldcg(p.kv_indptr + r), last = __ldcg(p.kv_indptr + r + 1);
      const int kvlen = (last - first - 1) * p.page_size + __ldcg(p.kv_last_page_len + r);
      for (int t = q0; t < q1; ++t) {
        tab.pos[t] = kvlen - (q1 - t);
        tab.kvb[t] = first;
        tab.req[t] = r;
        tab.fresh[t] = kvlen - (q1 - q0);
      }
    }
  }
  consumer_sync();
#pragma unroll 1
  for (int t = c.tid; t < T; t += kNumConsumers) {
    const int pos = tab.pos[t];
    tab.slot[t] = pos >= 0 ? (__ldcg(p.kv_indices + tab.kvb[t] + (pos >> p.page_shift)) << p.page_shift) + (pos & (p.page_size - 1)) : -1;
  }
  c.attn_iter = -1;
  consumer_sync();
}

// ------------------------------------------------------------------------------------
// the MMA issuer (one elected lane of warp 10)
// ------------------------------------------------------------------------------------
// Waits for the consumers to publish iteration `iter`; false: the launch ends.
__device__ __forceinline__ bool wait_go(const Ctx& c, volatile int* fl, int iter, int& go) {
  unsigned long long t0 = 0;
  int spins = 0;
  while (true) {
    go = fl[0];
    if (go < 0 || (go >> 8) >= iter) return go >= 0;
    __nanosleep(40);
    if (((++spins) & 255) == 0) {
      if (aborted(c)) return false;
      const unsigned long long now = globaltimer();
      if (t0 == 0) t0 = now;
      if (now - t0 > 4 * c.p.timeout_ns) return false;
    }
  }
}

// Waits until the consumers have counted linear op `seq` in flag word `word`; false: the launch ends.
__device__ __forceinline__ bool wait_lin(const Ctx& c, volatile int* fl, int word, unsigned seq) {
  unsigned long long t0 = 0;
  int spins = 0;
  while ((unsigned)fl[word] < seq) {
    if (fl[0] < 0) return false;
    __nanosleep(32);  // a hot spin would take issue slots from the consumer warps of this scheduler
    if (((++spins) & 1023) == 0) {
      if (aborted(c)) return false;
      const unsigned long long now = globaltimer();
      if (t0 == 0) t0 = now;
      if (now - t0 > 4 * c.p.timeout_ns) return false;
    }
  }
  return true;
}

// See WeightRing for the tiles that wait in tensor memory, 7 up to 32 token rows, 6 up to 64, 4 beyond.
__device__ __forceinline__ void mma_loop(Ctx& c) {
  const KParams& p = c.p;
  const int S = p.num_stages, N = p.x_rows;
  WeightRing ring(c, wide_slots(N), c.tmem + 2u * (uint32_t)N);
  volatile int* fl = c.flags();
  const uint32_t x_sub = (uint32_t)N * 128u;  // bytes of one activation box
  // instruction descriptor: D = f32, A = B = bf16, both K-major, N >> 3, M >> 4
  const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((128u >> 4) << 24);
  const int flying = N <= 32 ? 1 : 0;
  int xs = 0;  // next stage of activation boxes
  uint32_t xparity = 0;
  unsigned runs = 0;  // accumulator runs started
  bool dead = false;
  for (int iter = 1; !dead; ++iter) {
    int go;
    if (!wait_go(c, fl, iter, go)) break;
    for (int oi = 0; oi < p.num_ops && !dead; ++oi) {
      const OpDesc& op = p.ops[oi];
      if (op.type != OP_LINEAR) continue;
      unsigned total, t0, t1;
      int G;
      if (!wide_range(p, op, total, G, t0, t1)) continue;
      const int nkt = op.nkt;
      int kt = (int)(t0 % (unsigned)nkt);
      bool fresh = true;
      for (unsigned tile = t0; tile < t1; ++tile) {
        if ((fresh && !ring.wait(c.acc_empty_bar(runs & 1), ((runs >> 1) & 1u) ^ 1u)) || !ring.wait(c.xfull_bar(xs), xparity, flying) || !ring.wait_tile()) {
          dead = true;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t d = c.tmem + (runs & 1u) * (uint32_t)N, xt = c.xbox(xs);
        if (ring.held == 0) {  // straight from shared memory
          const uint32_t st = ring.stage();
#pragma unroll
          for (int sub = 0; sub < kSubTiles; ++sub) {
            const uint64_t ad = umma_smem_desc(st + (uint32_t)sub * kSubBytes);
            const uint64_t bd = umma_smem_desc(xt + (uint32_t)sub * x_sub);
#pragma unroll
            for (int k16 = 0; k16 < 4; ++k16)  // 16 k-elements = 32 bytes further inside the swizzle span: +2 in the address field
              umma_bf16(d, ad + (uint64_t)(2 * k16), bd + (uint64_t)(2 * k16), idesc, (fresh && sub == 0 && k16 == 0) ? 0u : 1u);
          }
          ring.free_stage();
        } else {
          const uint32_t at = ring.slot();
#pragma unroll
          for (int sub = 0; sub < kSubTiles; ++sub) {
            const uint64_t bd = umma_smem_desc(xt + (uint32_t)sub * x_sub);
#pragma unroll
            for (int k16 = 0; k16 < 4; ++k16)
              umma_bf16_ta(d, at + 32u * sub + 8u * k16, bd + (uint64_t)(2 * k16), idesc, (fresh && sub == 0 && k16 == 0) ? 0u : 1u);
          }
          ring.free_slot();
        }
        umma_commit(c.xempty_bar(xs));
        if (++xs == S) {
          xs = 0;
          xparity ^= 1u;
        }
        fresh = false;
        if (++kt == nkt || tile + 1 == t1) {  // the run ends: its accumulators belong to the finishing warps
          umma_commit(c.acc_full_bar(runs & 1));
          ++runs;
          fresh = true;
          kt = 0;
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

// ------------------------------------------------------------------------------------
// the input norm of a linear (F_NORM_IN)
// ------------------------------------------------------------------------------------
// A norm between two linears has no op of its own up to kNormBoxRows token rows: as one it is a barrier, a round trip and
// 3.6 us per norm at 8 requests of 8B width.  The linear before it stores the sums of squares of its output
// rows (F_ROW_SUMS), the consumers turn them into a scale per token at the start of the linear behind it while the first
// raw boxes are on their way, and warp 11 normalises every box in place: w * bf16(x * r) or x * (r * w), the arithmetic of
// the norm op.  Measured, us per step with a norm op and with the boxes, 12 layers: 8B width, 4 requests 1337 and 1267, 8 1353
// and 1290, 32 1535 and 1484; 2048 hidden, 8 requests 785 and 725; four layers of 1024 hidden, 4 requests 227 and 214.
__device__ __forceinline__ uint32_t hmul2_bf16(uint32_t a, uint32_t b) {  // both products rounded to bf16: exact in fp32 before that
  uint32_t d;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
// Scales of the iteration's tokens, by the consumers.  Warp w takes tokens w, w + 8, ...; op.ll_in: [token][ll_in_op] sums.
__device__ __forceinline__ void wide_row_scales(Ctx& c, const OpDesc& op, int T) {
  const bool torch_num = c.p.numerics == NUM_TORCH;
  const int parts = op.ll_in_op, nvec = parts >> 2;
  uint32_t* scale = wide_tab(c).scale;
  float ss[kNormBoxRows / kNumConsumerWarps];
#pragma unroll
  for (int i = 0; i < kNormBoxRows / kNumConsumerWarps; ++i) ss[i] = 0.f;
#pragma unroll 1
  for (int v = c.lane; v < nvec; v += 32) {
    float4 q[kNormBoxRows / kNumConsumerWarps];
#pragma unroll
    for (int i = 0; i < kNormBoxRows / kNumConsumerWarps; ++i) {
      const int t = c.warp + kNumConsumerWarps * i;
      q[i] = t < T ? __ldcg(reinterpret_cast<const float4*>(reinterpret_cast<const float*>(op.ll_in) + (size_t)t * parts) + v) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < kNormBoxRows / kNumConsumerWarps; ++i) ss[i] += (q[i].x + q[i].y) + (q[i].z + q[i].w);
  }
#pragma unroll
  for (int i = 0; i < kNormBoxRows / kNumConsumerWarps; ++i)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], o);
  // lane i finishes token w + 8 i (as row_rms_scale does for a staged row)
  float mine = ss[0];
#pragma unroll
  for (int i = 1; i < kNormBoxRows / kNumConsumerWarps; ++i) mine = c.lane == i ? ss[i] : mine;
  const int t = c.warp + kNumConsumerWarps * c.lane;
  if (t < T && c.lane < kNormBoxRows / kNumConsumerWarps) {
    const float r = torch_num ? torch_rsqrt_bf16(rbf(mine / (float)op.k), true) : rsqrtf(mine / (float)op.k + 1e-6f);
    scale[(t & 1) * (kNormBoxRows / 2) + (t >> 1)] = torch_num ? pack2(r, r) : __float_as_uint(r);
  }
  consumer_sync();
  if (c.tid == 0) {
    __threadfence_block();
    c.flags()[6] = (int)c.lin_seq;  // the norm warp may read them
  }
}

// The norm warp (warp 11).  Lane l holds 16-byte column l & 15 of a stage's two boxes for token rows (l >> 4), + 2, ...
// All it keeps has to fit the registers of a service warp, or spills sit in the loop that has to keep up with the weight stream.  With
// the 72 it has here four rows are in flight ("mpk", which unpacks them to fp32: two); with 56 it was half as many (32 requests 1520 us
// per step of 12 layers of 8B width instead of 1421).  Every lane arrives by itself: a __syncwarp in front of a single arrival costs
// registers in every loop around it.
__device__ __forceinline__ void norm_loop(Ctx& c) {
  const KParams& p = c.p;
  const int S = p.num_stages;
  volatile int* fl = c.flags();
  const int col = c.lane & 15, row0 = c.lane >> 4;
  // rows row0 + 2 u of eight: 256 u bytes further, in the 16-byte column that the swizzle gives them
  const uint32_t swz = (uint32_t)(((col & 7) ^ row0) << 4);
  const uint32_t sub = (uint32_t)(col >> 3) * (uint32_t)p.x_rows * 128u + (uint32_t)row0 * 128u;
  int s = 0;
  unsigned raw_phase = 0;  // per stage: parity of its next raw box
  unsigned lin_seq = 0;
  for (int iter = 1;; ++iter) {
    int go;
    if (!wait_go(c, fl, iter, go)) return;
    const int T = go & 255;
    for (int oi = 0; oi < p.num_ops; ++oi) {
      const OpDesc& op = p.ops[oi];
      if (op.type != OP_LINEAR) continue;
      lin_seq += 1;
      unsigned total, t0, t1;
      int G;
      if (!wide_range(p, op, total, G, t0, t1)) continue;
      if (!(op.flags & F_NORM_IN)) {  // (its boxes take the stages in turn all the same)
        s = (int)(((unsigned)s + (t1 - t0)) % (unsigned)S);
        continue;
      }
      // the weights of the first stages: they depend on nobody
      const uint4* nw = reinterpret_cast<const uint4*>(op.norm_w) + col;
      const int kvec = (op.k >> 3) - col, k_end = op.nkt * 16;  // (16 vectors of eight columns per tile)
      int kv = (int)(t0 % (unsigned)op.nkt) * 16;
      auto weights = [&](int k) { return k < kvec ? __ldg(nw + k) : make_uint4(0u, 0u, 0u, 0u); };
      uint4 w = weights(kv);
      if (!wait_lin(c, fl, 6, lin_seq)) return;
      __threadfence_block();
#pragma unroll 1
      for (int left = (int)(t1 - t0); left > 0; --left) {
        kv = kv + 16 == k_end ? 0 : kv + 16;
        const uint4 w_next = weights(kv);
        if (!mbar_wait(c, c.xraw_bar(s), (raw_phase >> s) & 1u, ST_TIMEOUT_FULL)) return;
        uint32_t box = c.xbox(s) + sub;
        uint32_t sc = smem_u32(wide_tab(c).scale) + (uint32_t)row0 * (kNormBoxRows / 2) * 4u;
        // (rows past T, still inside the box, are nobody's)
        if (p.numerics == NUM_TORCH) {
#pragma unroll 1
          for (int t = 0; t < T; t += 8) {
            uint4 x[4];
            const uint4 r = lds128(sc);
#pragma unroll
            for (int u = 0; u < 4; ++u) x[u] = lds128(box + 256u * u + (swz ^ (32u * u)));
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const uint32_t ru = u == 0 ? r.x : (u == 1 ? r.y : (u == 2 ? r.z : r.w));
              sts128(box + 256u * u + (swz ^ (32u * u)), make_uint4(hmul2_bf16(w.x, hmul2_bf16(x[u].x, ru)), hmul2_bf16(w.y, hmul2_bf16(x[u].y, ru)),
                                                                    hmul2_bf16(w.z, hmul2_bf16(x[u].z, ru)), hmul2_bf16(w.w, hmul2_bf16(x[u].w, ru))));
            }
            box += 1024;
            sc += 16;
          }
        } else {
#pragma unroll 1
          for (int t = 0; t < T; t += 8) {
#pragma unroll
            for (int u = 0; u < 4; u += 2) {
              const uint32_t at0 = box + 256u * u + (swz ^ (32u * u)), at1 = box + 256u * (u + 1) + (swz ^ (32u * (u + 1)));
              const uint4 x0 = lds128(at0), x1 = lds128(at1);
              const uint2 r = lds64(sc + 4 * u);
              sts128(at0, scale8(x0, w, __uint_as_float(r.x), false));
              sts128(at1, scale8(x1, w, __uint_as_float(r.y), false));
              if (u == 0 && t + 4 >= T) break;  // (rows t + 4 .. t + 7 are nobody's)
            }
            box += 1024;
            sc += 16;
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the tensor core reads the rows through the async proxy
        mbar_arrive(c.xfull_bar(s));
        raw_phase ^= 1u << s;
        if (++s == S) s = 0;
        w = w_next;
      }
    }
    if (p.mode == MODE_ONEPASS) return;
  }
}

// ------------------------------------------------------------------------------------
// finishing a run of tiles
// ------------------------------------------------------------------------------------
// Warp w reads accumulator lanes 32 (w & 3) .. + 31 (weight rows of the tile) and one half of the token columns;
// a thread holds one output row for up to 32 tokens in registers, from tensor memory to the store.
//
// Several CTAs hold k-ranges of a row block; their sums are added up in CTA order.  No CTA-wide sync and no shared memory on the way.
//  * A block is finished by the CTA with its FIRST k-range (that range is the tail of its own tile range, so it is computed last
//    anyway), or, where there are few blocks (wide_shares), by all of its CTAs, each a share of the tokens, behind the op's last tile: one
//    CTA would read up to six pieces and more in turn, 5 to 7 us of a linear's end.
//  * Up to 32 token rows (linear_wide) sums travel as words that carry a tag, two tokens per 16 bytes, [token / 2][row], and
//    a finishing thread polls those of its own output row, several pieces at once: data and "ready" arrive in one load, with no
//    release behind the stores, no flag and no second round trip.  The tag differs in every op of every iteration, the words are
//    cleared before every launch, and a CTA's slot is written again only behind a grid barrier.
//  * Beyond (linear_wide_shared), twice the bytes cost more than the round trip: plain float4 of four tokens, [token / 4][row]; every
//    warp publishes its share with a release of its own, a flag that holds the op's tag, for the matching warps of the other CTAs.
// 12 layers of 8B width, us per step with one finishing CTA per block and with shares: 64 requests 1671 and 1573, 100 2193 and
// 2053; 17 1324 and 1294, 32 1400 and 1391; 2048 hidden, 32 requests 890 and 811.
__device__ __forceinline__ uint32_t order_bf16(float v) {  // monotone 16-bit key of a bf16 value; 0 only for NaN
  const uint32_t b = __float_as_uint(v + 0.f) >> 16;       // (-0 counts as +0)
  const uint32_t k = (b & 0x8000u) ? (~b & 0xffffu) : (b | 0x8000u);
  return v != v ? 0u : k;
}
__device__ __forceinline__ float unorder_bf16(uint32_t k) {
  const uint32_t b = (k & 0x8000u) ? (k & 0x7fffu) : (~k & 0xffffu);
  return __uint_as_float(b << 16);
}
// running best logit per token of a warp's rows: lane i holds token column c0 + i
struct WideBest {
  uint32_t key[2];
  int idx[2];
};

// The q/k/v head vector of a token, 8 dims per lane of a half-warp: RMSNorm + RoPE for q and k, then q goes to the
// attention's scratch rows and k / v to their cache row.  `part`: q head (< qpk), qpk = k, qpk + 1 = v.
__device__ __forceinline__ void wide_store_head(const Ctx& c, const OpDesc& op, uint4 raw, int tok, int h, int part, bool live, int l16) {
  const KParams& p = c.p;
  const int HKV = op.aux0, qpk = op.aux1 / op.aux0;
  const WideTab& tab = wide_tab(c);
  uint4 y = raw;
  if (__any_sync(0xffffffffu, part <= qpk)) {  // (the halves of a warp may hold different parts: the shuffles below want both)
    const int pos = min(max(tab.pos[tok], 0), op.aux2 - 1);  // aux2 = rows of the cos/sin tables
    const uint4 w = __ldg(reinterpret_cast<const uint4*>(part < qpk ? op.q_norm_w : op.k_norm_w) + l16);
    const uint4 cs = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(op.cos) + (size_t)pos * kHeadDim) + l16);
    const uint4 sn = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(op.sin) + (size_t)pos * kHeadDim) + l16);
    F8 f;
    unpack8(raw, f.v);
    f = head_norm_rope(f, w, cs, sn, l16, op.aux3, p.numerics, part < qpk ? op.aux1 < 32 : op.aux0 < 32);
    if (part <= qpk) y = pack8(f.v);
  }
  if (!live) return;
  if (part < qpk) {
    reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(op.out2) + (size_t)tok * op.ld_out2 + (size_t)(h * qpk + part) * kHeadDim)[l16] = y;
  } else {
    const int slot = tab.slot[tok];
    if (slot < 0) return;
    __nv_bfloat16* cache = reinterpret_cast<__nv_bfloat16*>(part == qpk ? op.k_cache : op.v_cache);
    reinterpret_cast<uint4*>(cache + ((size_t)slot * HKV + h) * kHeadDim)[l16] = y;
  }
}

// `cc`, `l0`: where the running best of the first token is kept (pair, lane)
template <int NC>
__device__ __forceinline__ void wide_epilogue(Ctx& c, const OpDesc& op, int blk, int row, int tok0, int nlive, const float (&v)[NC],
                                              const uint32_t (&res)[NC / 2], WideBest& best, int cc = 0, int l0 = 0) {
  constexpr bool kSums = 2 * MK_NC <= kNormBoxRows;
  const KParams& p = c.p;
  const int col = blk * kTileRows + row;
  __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(op.out);
  if (op.flags & F_SILU_MUL) {
    // weight rows are units of [4 gate | 4 up]: lanes l and l ^ 4 hold the two halves of four output columns.  Of
    // every pair of tokens the gate lane finishes the even one, the up lane the odd one.
    const bool up = (row & 4) != 0;
    const int ocol = blk * 64 + (row >> 3) * 4 + (row & 3);
    const bool okc = ocol < (op.n >> 1);
#pragma unroll
    for (int i = 0; i < NC; i += 2) {
      const float mine0 = rbf(v[i]), mine1 = rbf(v[i + 1]);  // the linear output is bf16 before the activation
      const float other = __shfl_xor_sync(0xffffffffu, up ? mine0 : mine1, 4);
      const float g = up ? other : mine0, u = up ? mine1 : other;
      const float y = rbf(__fdividef(g, 1.0f + __expf(-g))) * u;
      const int t = i + (up ? 1 : 0);
      if (okc && t < nlive) out[(size_t)(tok0 + t) * op.ld_out + ocol] = __float2bfloat16_rn(y);
    }
    return;
  }
  if (op.flags & F_QKV_PREP) {
    // a row block is one head vector of every token: transposed through shared memory (16 token rows per column
    // half and round), then a half-warp per token.  The four warps of a half meet on a named barrier of their own.
    const int half = c.warp >> 2, q = c.warp & 3, l16 = c.lane & 15;
    const int qpk = op.aux1 / op.aux0;
    constexpr int kRound = NC < 16 ? NC : 16;
    __nv_bfloat16* buf = reinterpret_cast<__nv_bfloat16*>(c.smem + p.x_off) + half * kRound * kHeadDim;
#pragma unroll
    for (int c0 = 0; c0 < NC; c0 += kRound) {
#pragma unroll
      for (int i = 0; i < kRound; ++i) buf[i * kHeadDim + row] = __float2bfloat16_rn(v[c0 + i]);
      asm volatile("bar.sync %0, 128;" ::"r"(2 + half) : "memory");
#pragma unroll 1
      for (int t = q * 2 + (c.lane >> 4); t < kRound; t += 8)
        wide_store_head(c, op, reinterpret_cast<const uint4*>(buf + t * kHeadDim)[l16], tok0 + (c0 + t < nlive ? c0 + t : 0), blk / (qpk + 2),
                        blk % (qpk + 2), c0 + t < nlive, l16);
      asm volatile("bar.sync %0, 128;" ::"r"(2 + half) : "memory");
    }
    return;
  }
  const bool okc = col < op.n;
  const bool push = MK_XF(op, F_PUSH) != 0;
  const bool with_res = (op.flags & F_RESIDUAL) && (!(op.flags & F_RES_RANK0) || p.rank == 0);
  float sq[kSums ? NC : 1];
  const bool rnd = p.numerics == NUM_TORCH && !push;  // (pushed partial sums stay fp32: rounded once, after the ranks are added up)
#pragma unroll
  for (int i = 0; i < NC; ++i) {
    float y = v[i];
    if (with_res) {
      float r = (i & 1) ? bf_hi(res[i >> 1]) : bf_lo(res[i >> 1]);
      if (MK_XF(op, F_GATHER_RES) && okc && i < nlive) r = xchg_gather1(c, xchg_cur(c), tok0 + i, col);
      y = (rnd ? rbf(y) : y) + r;
    }
    if (okc && i < nlive) {
      if (push) xchg_push1(p, xchg_next(c), tok0 + i, col, y);
      else out[(size_t)(tok0 + i) * op.ld_out + col] = __float2bfloat16_rn(y);
    }
    if constexpr (kSums) {
      y = okc ? rbf(y) : 0.f;
      sq[i] = p.numerics == NUM_TORCH ? rbf(y * y) : y * y;
    }
  }
  if constexpr (kSums) {
    if (op.flags & F_ROW_SUMS) {
      // NC sums over the warp's 32 rows: halves change places until a lane is left with one token, then the rest is added up
      int tok = 0;
#pragma unroll
      for (int n = NC, o = 16; n > 1; n >>= 1, o >>= 1) {
        const bool upper = (c.lane & o) != 0;
#pragma unroll
        for (int i = 0; i < n / 2; ++i) {
          const float give = upper ? sq[i] : sq[i + n / 2];
          sq[i] = (upper ? sq[i + n / 2] : sq[i]) + __shfl_xor_sync(0xffffffffu, give, o);
        }
        if (upper) tok += n / 2;
      }
#pragma unroll
      for (int o = 16 / NC; o > 0; o >>= 1) sq[0] += __shfl_xor_sync(0xffffffffu, sq[0], o);
      if ((c.lane & (32 / NC - 1)) == 0 && tok < nlive)
        reinterpret_cast<float*>(op.ll_out)[(size_t)(tok0 + tok) * (size_t)op.ll_res_op + blk * 4 + (row >> 5)] = sq[0];
    }
  }
  if (op.flags & F_ARGMAX) {
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      // larger value wins, ties go to the lower index: one 32-bit maximum over the warp's rows
      const uint32_t k = okc ? (order_bf16(rbf(v[i])) << 16) | (uint32_t)(0xffff - row) : 0u;
      const uint32_t m = __reduce_max_sync(0xffffffffu, k);
      // (an equal value keeps the lower index; indexed by cc, the pairs would live in local memory)
      const uint32_t key = m >> 16, had = cc == 0 ? best.key[0] : best.key[1];
      const int at = blk * kTileRows + 0xffff - (int)(m & 0xffffu);
      if (c.lane == l0 + i && key != 0u && (key > had || (key == had && at < (cc == 0 ? best.idx[0] : best.idx[1])))) {
        if (cc == 0) {
          best.key[0] = key;
          best.idx[0] = at;
        } else {
          best.key[1] = key;
          best.idx[1] = at;
        }
      }
    }
  }
}

// The residual of NC tokens from col0 on, pairs of bf16 (zeros where there is none)
template <int NC>
__device__ __forceinline__ void wide_residual(const OpDesc& op, bool with_res, int col, int col0, int nlive, uint32_t (&res)[NC / 2]) {
#pragma unroll
  for (int i = 0; i < NC / 2; ++i) res[i] = 0u;
  if (!with_res || col >= op.n) return;
  const unsigned short* rp = reinterpret_cast<const unsigned short*>(op.res) + (size_t)col0 * op.ld_res + col;
#pragma unroll
  for (int i = 0; i < NC / 2; ++i) {
    uint32_t lo = 0u, hi = 0u;
    if (2 * i < nlive) lo = __ldcg(rp + (size_t)(2 * i) * op.ld_res);
    if (2 * i + 1 < nlive) hi = __ldcg(rp + (size_t)(2 * i + 1) * op.ld_res);
    res[i] = lo | (hi << 16);
  }
}
__device__ __forceinline__ bool wide_with_res(const Ctx& c, const OpDesc& op) {
  return (op.flags & F_RESIDUAL) && !MK_XF(op, F_GATHER_RES) && (!(op.flags & F_RES_RANK0) || c.p.rank == 0);
}
// The live token columns are split evenly over the two halves of the warps: the upper half's first column.  In steps of the two
// tokens of a word, beyond 32 token rows of the eight that a share is made of.
template <int NC>
__device__ __forceinline__ int wide_split(int T) {
  constexpr int step = NC < 32 ? 2 : 8;
  return (T + 2 * step - 1) / (2 * step) * step;
}
// one (max, index) partial per token, CTA and row quarter; NC token columns per pair of `best`
template <int NC>
__device__ __forceinline__ void wide_store_best(const Ctx& c, const OpDesc& op, int T, int G, int pairs, const WideBest& best) {
#pragma unroll
  for (int cc = 0; cc < 2; ++cc) {
    const int half = c.warp >> 2, t0 = wide_split<NC>(T), t = half * t0 + cc * NC + c.lane;
    if (cc < pairs && c.lane < NC && t < (half == 0 ? min(t0, T) : T) && (int)blockIdx.x < G) {
      const size_t o = (size_t)t * op.amax_n + blockIdx.x * 4 + (c.warp & 3);
      op.amax_val[o] = best.key[cc] != 0u ? unorder_bf16(best.key[cc]) : -INFINITY;
      op.amax_idx[o] = best.idx[cc];
    }
  }
}

// Up to 32 token rows: where a piece of a block lies.  A CTA has two slots: the block its range begins in, and the one it ends in.
__device__ __forceinline__ uint4* wide_words(const KParams& p, int cta, int slot) {
  return p.partial + ((size_t)cta * 2 + slot) * (size_t)(kTileRows * p.x_rows / 2);
}
// This CTA's share of a block's tokens: of the groups of NC / 4 tokens of each half, as many as there are CTAs to share them, in CTA
// order.
template <int NC>
__device__ __forceinline__ void wide_finish_words(Ctx& c, const OpDesc& op, int T, int blk, unsigned total, int G, WideBest& best) {
  constexpr int NT = NC / 4;
  const KParams& p = c.p;
  const int half = c.warp >> 2, row = 32 * (c.warp & 3) + c.lane, col = blk * kTileRows + row;
  const unsigned blk0 = (unsigned)blk * (unsigned)op.nkt;
  const int c_first = tile_owner(blk0, total, G), P = tile_owner(blk0 + (unsigned)op.nkt - 1u, total, G) - c_first + 1, me = (int)blockIdx.x - c_first;
  const int split = wide_split<NC>(T), end = half == 0 ? min(split, T) : T;
  const int groups = max(0, (end - half * split + NT - 1) / NT);
  const int g0 = (me * groups + P - 1) / P, g1 = ((me + 1) * groups + P - 1) / P;
  if (g0 >= g1) return;  // (the same in all four warps of a half)
  const unsigned tag = ll_tag_of(c, c.cur_op);
  const int slot = tile_begin((unsigned)c_first, total, (unsigned)G) == blk0 ? 0 : 1;  // of the first piece; the others open their CTA's range
  const bool with_res = wide_with_res(c, op);
#pragma unroll 1
  for (int g = g0; g < g1; ++g) {
    const int tok0 = half * split + NT * g, nlive = min(NT, end - tok0);
    uint32_t res[NT / 2];
    wide_residual<NT>(op, with_res, col, tok0, nlive, res);  // (does not depend on the sums: requested first)
    float v[NT];
#pragma unroll
    for (int i = 0; i < NT; ++i) v[i] = 0.f;
    constexpr int PB = 6;  // pieces in flight per round
#pragma unroll 1
    for (int i0 = 0; i0 < P; i0 += PB) {
      uint4 w[PB][NT / 2];
#pragma unroll
      for (int u = 0; u < PB; ++u)
#pragma unroll
        for (int i = 0; i < NT / 2; ++i) {
          const unsigned t = (i0 + u < P && 2 * i < nlive) ? ~tag : tag;  // (nothing to wait for: zeros)
          w[u][i] = make_uint4(0u, t, 0u, t);
        }
      PollLimit limit;
      while (true) {
#pragma unroll
        for (int u = 0; u < PB; ++u)
#pragma unroll
          for (int i = 0; i < NT / 2; ++i)
            if (w[u][i].y != tag || w[u][i].w != tag)
              w[u][i] = ld_gpu_words(wide_words(p, c_first + i0 + u, i0 + u == 0 ? slot : 0) + (size_t)((tok0 >> 1) + i) * kTileRows + row);
        bool here = true;
#pragma unroll
        for (int u = 0; u < PB; ++u)
#pragma unroll
          for (int i = 0; i < NT / 2; ++i) here = here && w[u][i].y == tag && w[u][i].w == tag;
        if (here || limit.expired(c, tag, w[0][0].y)) break;
      }
#pragma unroll
      for (int u = 0; u < PB; ++u)
#pragma unroll
        for (int i = 0; i < NT / 2; ++i) {
          v[2 * i] += __uint_as_float(w[u][i].x);
          v[2 * i + 1] += __uint_as_float(w[u][i].z);
        }
    }
    __syncwarp();  // (lanes leave the poll at different times; the epilogue shuffles)
    wide_epilogue<NT>(c, op, blk, row, tok0, nlive, v, res, best, 0, NT * g);
  }
}
// NC: token columns of a thread, x_rows / 2
template <int NC>
__device__ __forceinline__ void linear_wide(Ctx& c, const OpDesc& op, int T) {
  const KParams& p = c.p;
  const int N = p.x_rows, nkt = op.nkt;
  const int q = c.warp & 3, half = c.warp >> 2, row = 32 * q + c.lane;
  WideBest best;
  best.key[0] = best.key[1] = 0u;
  best.idx[0] = best.idx[1] = 0x7fffffff;
  unsigned total, t0, t1;
  int G;
  if (wide_range(p, op, total, G, t0, t1)) {
    const bool with_res = wide_with_res(c, op), share = wide_shares(op, G, N, T);
    int shared[2] = {-1, -1};  // blocks to finish with others: the one the range begins in, the one it ends in
    const unsigned tag = ll_tag_of(c, c.cur_op);
    const int col0 = half * wide_split<NC>(T);  // first token column of this thread
    const int nlive = half == 0 ? min(wide_split<NC>(T), T) : T - col0;  // may be none: nothing but padding
#pragma unroll 1
    for (unsigned tile = t0; tile < t1;) {
      const int blk = (int)(tile / (unsigned)nkt);
      const unsigned blk0 = (unsigned)blk * (unsigned)nkt, blk1 = blk0 + (unsigned)nkt;
      const int c_last = tile_owner(blk1 - 1, total, G);
      const bool first = tile == t0, finisher = tile == blk0 && (!share || c_last == (int)blockIdx.x);
      const uint32_t acc = c.tmem + (c.acc_runs & 1u) * (uint32_t)N + ((uint32_t)(32 * q) << 16);
      // the residual does not depend on the sums: requested first
      uint32_t res[NC / 2];
      wide_residual<NC>(op, with_res && finisher, blk * kTileRows + row, col0, nlive, res);
      mbar_wait(c, c.acc_full_bar(c.acc_runs & 1), (c.acc_runs >> 1) & 1u, ST_TIMEOUT_FULL);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (first) MK_STAMP(c, 0);
      __syncwarp();
      uint32_t raw[NC];
      tmem_ld<NC>(acc + (uint32_t)col0, raw);
      tmem_wait_ld();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (c.lane == 0) mbar_arrive(c.acc_empty_bar(c.acc_runs & 1));  // the accumulators may be overwritten
      c.acc_runs += 1;
      tile = min(blk1, t1);
      float v[NC];
#pragma unroll
      for (int i = 0; i < NC; ++i) v[i] = __uint_as_float(raw[i]);
      if (!finisher) {
        uint4* mine = wide_words(p, (int)blockIdx.x, first ? 0 : 1) + (size_t)(col0 >> 1) * kTileRows + row;
#pragma unroll
        for (int i = 0; i < NC / 2; ++i)
          if (2 * i < nlive) st_gpu_words(mine + (size_t)i * kTileRows, __float_as_uint(v[2 * i]), __float_as_uint(v[2 * i + 1]), tag);
        if (share) (first ? shared[0] : shared[1]) = blk;
        MK_STAMP(c, 1);
        continue;
      }
      MK_STAMP(c, 2);
      if (c_last > (int)blockIdx.x) {
        const uint4* src0 = wide_words(p, 0, 0) + (size_t)(col0 >> 1) * kTileRows + row;
        const size_t stride = (size_t)(wide_words(p, 1, 0) - wide_words(p, 0, 0));
        // Several pieces in flight per round (registers allowing): a block of a small layer has up to `nkt` of them.
        constexpr int PB = NC == 8 ? 4 : 2;
#pragma unroll 1
        for (int cta = (int)blockIdx.x + 1; cta <= c_last; cta += PB) {
          uint4 w[PB][NC / 2];
#pragma unroll
          for (int u = 0; u < PB; ++u)
#pragma unroll
            for (int i = 0; i < NC / 2; ++i) {
              const unsigned t = (cta + u <= c_last && 2 * i < nlive) ? ~tag : tag;  // (nothing to wait for: zeros)
              w[u][i] = make_uint4(0u, t, 0u, t);
            }
          PollLimit limit;
          while (true) {
#pragma unroll
            for (int u = 0; u < PB; ++u)
#pragma unroll
              for (int i = 0; i < NC / 2; ++i)
                if (w[u][i].y != tag || w[u][i].w != tag) w[u][i] = ld_gpu_words(src0 + (size_t)(cta + u) * stride + (size_t)i * kTileRows);
            bool here = true;
#pragma unroll
            for (int u = 0; u < PB; ++u)
#pragma unroll
              for (int i = 0; i < NC / 2; ++i) here = here && w[u][i].y == tag && w[u][i].w == tag;
            if (here || limit.expired(c, tag, w[0][0].y)) break;
          }
#pragma unroll
          for (int u = 0; u < PB; ++u)
#pragma unroll
            for (int i = 0; i < NC / 2; ++i) {
              v[2 * i] += __uint_as_float(w[u][i].x);
              v[2 * i + 1] += __uint_as_float(w[u][i].z);
            }
        }
        MK_STAMP(c, 3);
      }
      __syncwarp();  // (lanes leave the poll at different times; the epilogue shuffles)
      MK_STAMP(c, 4);
      wide_epilogue<NC>(c, op, blk, row, col0, nlive, v, res, best);
      MK_STAMP(c, 5);
    }
    // the block the range ends in first: its other CTAs began with it
#pragma unroll 1
    for (int i = 1; i >= 0; --i) {
      const int blk = i == 1 ? shared[1] : shared[0];
      if (blk >= 0) wide_finish_words<NC>(c, op, T, blk, total, G, best);
    }
    MK_STAMP(c, 6);
  }
  if (op.flags & F_ARGMAX) wide_store_best<NC>(c, op, T, G, 1, best);
}

// Beyond 32 token rows: where a piece of a block lies.  A CTA has two slots: the block its range begins in, and the one it ends in.
__device__ __forceinline__ float4* wide_piece(const KParams& p, int cta, int slot) {
  return reinterpret_cast<float4*>(p.partial) + ((size_t)cta * 2 + slot) * (size_t)(kTileRows * p.x_rows / 4);
}
__device__ __forceinline__ unsigned* wide_flag(const KParams& p, int cta, int slot) { return p.piece_flag + ((size_t)cta * 2 + slot) * kNumConsumerWarps; }
// Waits until the matching warps of CTAs c0 .. c1 have published their pieces; `slot`: the one of c0 (the others open their ranges).
__device__ __forceinline__ void wide_wait_pieces(const Ctx& c, int c0, int c1, int slot, unsigned tag) {
  for (int cta = c0 + c.lane; cta <= c1; cta += 32) {
    const unsigned* flag = wide_flag(c.p, cta, cta == c0 ? slot : 0) + c.warp;
    PollLimit limit;
    unsigned got;
    while ((got = ld_acquire_u32(flag)) != tag && !limit.expired(c, tag, got, ST_TIMEOUT_PEER)) {
    }
  }
  __syncwarp();
}
// This CTA's share of a block's tokens: of the eight-token groups of each half, as many as there are CTAs to share them, in CTA order.
__device__ __forceinline__ void wide_finish_share(Ctx& c, const OpDesc& op, int T, int blk, unsigned total, int G, WideBest& best) {
  const KParams& p = c.p;
  const int half = c.warp >> 2, row = 32 * (c.warp & 3) + c.lane, col = blk * kTileRows + row;
  const unsigned blk0 = (unsigned)blk * (unsigned)op.nkt;
  const int c_first = tile_owner(blk0, total, G), P = tile_owner(blk0 + (unsigned)op.nkt - 1u, total, G) - c_first + 1, me = (int)blockIdx.x - c_first;
  const int split = wide_split<32>(T), end = half == 0 ? min(split, T) : T;
  const int groups = max(0, (end - half * split + 7) >> 3);
  const int g0 = (me * groups + P - 1) / P, g1 = ((me + 1) * groups + P - 1) / P;
  if (g0 >= g1) return;  // (the same in all four warps of a half)
  const unsigned tag = ll_tag_of(c, c.cur_op);
  const int slot = tile_begin((unsigned)c_first, total, (unsigned)G) == blk0 ? 0 : 1;  // of the first piece; the others open their CTA's range
  const bool with_res = wide_with_res(c, op);
#pragma unroll 1
  for (int g = g0; g < g1; ++g) {
    const int tok0 = half * split + 8 * g, nlive = min(8, end - tok0);
    uint32_t res[4];
    wide_residual<8>(op, with_res, col, tok0, nlive, res);  // (does not depend on the sums: requested first)
    if (g == g0) wide_wait_pieces(c, c_first, c_first + P - 1, slot, tag);
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = 0.f;
    constexpr int PB = 4;  // pieces in flight per round
#pragma unroll 1
    for (int i0 = 0; i0 < P; i0 += PB) {
      float4 w[PB][2];
#pragma unroll
      for (int u = 0; u < PB; ++u) {
        const int i = min(i0 + u, P - 1);
        const float4* src = wide_piece(p, c_first + i, i == 0 ? slot : 0) + (size_t)(tok0 >> 2) * kTileRows + row;
        w[u][0] = i0 + u < P ? __ldcg(src) : make_float4(0.f, 0.f, 0.f, 0.f);
        w[u][1] = i0 + u < P && nlive > 4 ? __ldcg(src + kTileRows) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int u = 0; u < PB; ++u)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          v[4 * i] += w[u][i].x;
          v[4 * i + 1] += w[u][i].y;
          v[4 * i + 2] += w[u][i].z;
          v[4 * i + 3] += w[u][i].w;
        }
    }
    wide_epilogue<8>(c, op, blk, row, tok0, nlive, v, res, best, g >> 2, 8 * (g & 3));
  }
}
__device__ __forceinline__ void linear_wide_shared(Ctx& c, const OpDesc& op, int T) {
  constexpr int NC = 32;  // token columns of a thread per round (128 token rows: two rounds)
  const KParams& p = c.p;
  const int N = p.x_rows, nkt = op.nkt, split = wide_split<NC>(T), nround = split > NC ? 2 : 1;
  const int q = c.warp & 3, half = c.warp >> 2, row = 32 * q + c.lane;
  WideBest best;
  best.key[0] = best.key[1] = 0u;
  best.idx[0] = best.idx[1] = 0x7fffffff;
  unsigned total, t0, t1;
  int G;
  if (wide_range(p, op, total, G, t0, t1)) {
    const bool with_res = wide_with_res(c, op), share = wide_shares(op, G, N, T);
    const unsigned tag = ll_tag_of(c, c.cur_op);
    int shared[2] = {-1, -1};  // blocks to finish with others: the one the range begins in, the one it ends in
#pragma unroll 1
    for (unsigned tile = t0; tile < t1;) {
      const int blk = (int)(tile / (unsigned)nkt);
      const unsigned blk0 = (unsigned)blk * (unsigned)nkt, blk1 = blk0 + (unsigned)nkt;
      const bool first = tile == t0, begins = tile == blk0;
      const int c_last = tile_owner(blk1 - 1, total, G);
      const bool finisher = begins && (!share || c_last == (int)blockIdx.x);
      const uint32_t acc = c.tmem + (c.acc_runs & 1u) * (uint32_t)N + ((uint32_t)(32 * q) << 16);
#pragma unroll 1
      for (int cc = 0; cc < nround; ++cc) {
        const int col0 = half * split + cc * NC;  // first token column of this thread's round
        const int nlive = min(NC, (half == 0 ? min(split, T) : T) - col0);  // may be none or less: nothing but padding
        // the residual does not depend on the sums: requested first
        uint32_t res[NC / 2];
        wide_residual<NC>(op, with_res && finisher, blk * kTileRows + row, col0, nlive, res);
        if (cc == 0) {
          mbar_wait(c, c.acc_full_bar(c.acc_runs & 1), (c.acc_runs >> 1) & 1u, ST_TIMEOUT_FULL);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
        if (first) MK_STAMP(c, 0);
        __syncwarp();
        uint32_t raw[NC];
        tmem_ld<NC>(acc + (uint32_t)col0, raw);
        tmem_wait_ld();
        if (cc == nround - 1) {  // the accumulators may be overwritten
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (c.lane == 0) mbar_arrive(c.acc_empty_bar(c.acc_runs & 1));
        }
        float v[NC];
#pragma unroll
        for (int i = 0; i < NC; ++i) v[i] = __uint_as_float(raw[i]);
        if (!finisher) {
          float4* mine = wide_piece(p, (int)blockIdx.x, first ? 0 : 1) + (size_t)(col0 >> 2) * kTileRows + row;
#pragma unroll
          for (int i = 0; i < NC / 4; ++i)
            if (4 * i < nlive) mine[(size_t)i * kTileRows] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
          if (cc == nround - 1) {
            __syncwarp();  // lane 0's release covers what the warp wrote before
            if (c.lane == 0)
              asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(wide_flag(p, (int)blockIdx.x, first ? 0 : 1) + c.warp), "r"(tag) : "memory");
            if (share) (first ? shared[0] : shared[1]) = blk;
          }
          if (first) MK_STAMP(c, 1);
          continue;
        }
        MK_STAMP(c, 2);
        if (c_last > (int)blockIdx.x) {
          if (cc == 0) wide_wait_pieces(c, (int)blockIdx.x + 1, c_last, 0, tag);
          const float4* src0 = wide_piece(p, 0, 0) + (size_t)(col0 >> 2) * kTileRows + row;
          const size_t stride = (size_t)kTileRows * N / 2;  // from a CTA's first piece to the next one's
          constexpr int PB = 2;  // pieces in flight per round
#pragma unroll 1
          for (int cta = (int)blockIdx.x + 1; cta <= c_last; cta += PB) {
            float4 w[PB][NC / 4];
#pragma unroll
            for (int u = 0; u < PB; ++u)
#pragma unroll
              for (int i = 0; i < NC / 4; ++i)
                w[u][i] = (cta + u <= c_last && 4 * i < nlive) ? __ldcg(src0 + (size_t)(cta + u) * stride + (size_t)i * kTileRows)
                                                               : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int u = 0; u < PB; ++u)
#pragma unroll
              for (int i = 0; i < NC / 4; ++i) {
                v[4 * i] += w[u][i].x;
                v[4 * i + 1] += w[u][i].y;
                v[4 * i + 2] += w[u][i].z;
                v[4 * i + 3] += w[u][i].w;
              }
          }
          MK_STAMP(c, 3);
        }
        __syncwarp();
        MK_STAMP(c, 4);
        wide_epilogue<NC>(c, op, blk, row, col0, nlive, v, res, best, cc);
        MK_STAMP(c, 5);
      }
      c.acc_runs += 1;
      tile = min(blk1, t1);
    }
    // the block the range ends in first: its other CTAs began with it
#pragma unroll 1
    for (int i = 1; i >= 0; --i) {
      const int blk = i == 1 ? shared[1] : shared[0];
      if (blk >= 0) wide_finish_share(c, op, T, blk, total, G, best);
    }
    MK_STAMP(c, 6);
  }
  if (op.flags & F_ARGMAX) wide_store_best<NC>(c, op, T, G, nround, best);
}

template <int NC>
__device__ __forceinline__ void op_linear_wide(Ctx& c, const OpDesc& op, int T) {
  if (op_barrier(c, op)) return;
  c.lin_seq += 1;
  if (c.tid == 0) c.flags()[4] = (int)c.lin_seq;  // the activation producer may now read this op's input
  if constexpr (2 * NC <= kNormBoxRows) {
    if (op.flags & F_NORM_IN) wide_row_scales(c, op, T);
  }
  if constexpr (2 * NC <= kNormBoxRows) linear_wide<NC>(c, op, T);
  else linear_wide_shared(c, op, T);
  if (MK_XF(op, F_PUSH)) c.ar_seq += 1;  // every CTA counts the exchange, with or without rows of its own
}

// ------------------------------------------------------------------------------------
// attention: paged GQA on the warp-level tensor cores
// ------------------------------------------------------------------------------------
// When this runs, the new tokens' K/V rows are in the cache and the normalised, rotated q rows in the op's scratch
// (stored by the QKV linear's epilogue, F_QKV_PREP, or by attn_prepare_rows below).
//
// A query group is up to 8 / qpk consecutive tokens of one request: with the q heads of a kv head they fill eight rows, so
// a prompt chunk reads a K/V row once per group instead of once per token (a decoding request is a group of one).  A task
// is (query group, kv head[, chunk of positions]); W = 1, 2, 4 or 8 warps share a task and take its 16-position tiles in
// turn:
//   S = Q K^T       mma.m16n8k16, M = the group's rows (eight of 16), N = 8 positions, K = 128 dims in 8 steps
//   O^T += V^T P^T  M = 16 dims in 8 tiles, N = the rows, K = 16 positions: the scores are its B operand as they are
// with the fragments loaded straight from the cache rows, no staging and no ldmatrix: a dot product does not care in
// which order the dims are walked, so k step s of lane j of a quad stands for dims 32 (s / 2) + 8 j + 4 (s % 2) +
// {0..3} (the quad reads 64 contiguous bytes of a K row per load), and rows n and n + 8 of dim tile t stand for dims
// 8 n + t and 64 + 8 n + t (eight lanes read 128 contiguous bytes of a V row per load; two rows are paired up per
// register with byte permutes).  P enters as the sum of three bf16 values (24 bits: what fp32 holds), and a score is
// the sum of two chains of four mma (a chain truncates what it adds up).  Outputs that are not the bf16 nearest to a
// float64 softmax, 4 to 40 requests: 0.038 %, the same as with scalar fp32; with one chain 0.040 %, with P as two bf16
// values 0.2 %, as one 10 to 34 %.  Two more mma per tile column cost nothing that could be measured.
// (Groups of 16 rows, with the rows on M in both products, took 64 registers of sums, half of them idle in decoding, and
// did not fit beside the other kind of group without 280 bytes of spills per thread.)
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}

struct WideTask {
  int t0, nt, h, ch, nch;  // first token, tokens, kv head, chunk, chunks
  int p0, p1, L0, kvb;     // positions [p0, p1) of this chunk; length the first token sees; page-table base
  int fresh;               // first position whose row this iteration writes
};

// Query groups, warps per task and chunking of the iteration: the same in every layer, worked out by the first
// attention op (key: the head geometry).
__device__ __forceinline__ void wide_plan_attention(Ctx& c, const OpDesc& op, int T) {
  const KParams& p = c.p;
  WideTab& tab = wide_tab(c);
  const int HKV = op.aux0, qpk = op.aux1 / op.aux0, tpg = 8 / qpk;
  T = min(T, kWideTab);
  // a token opens a group when it is the first of its request or tpg tokens behind the last opening
  int lmax = 1;
  bool opens = false;
  int first = 0, len = 0;
  if (c.tid < T) {
    const int r = tab.req[c.tid];
    first = __ldcg(p.qo_indptr + r);
    const int q1 = min(__ldcg(p.qo_indptr + r + 1), T);
    opens = (c.tid - first) % tpg == 0;
    len = min(tpg, q1 - c.tid);
    lmax = tab.pos[c.tid] + 1;
  }
  const unsigned bal = __ballot_sync(0xffffffffu, opens);
  const int wmax = __reduce_max_sync(0xffffffffu, lmax);
  if (c.lane == 0 && c.warp < 4) {
    tab.scan[c.warp] = __popc(bal);
    tab.scan[4 + c.warp] = wmax;
  }
  consumer_sync();
  if (opens) {
    int g = __popc(bal & ((1u << c.lane) - 1u));
    for (int w = 0; w < c.warp; ++w) g += tab.scan[w];
    tab.grp[g] = c.tid | (len << 8);
  }
  if (c.tid == 0) {
    const int ng = tab.scan[0] + tab.scan[1] + tab.scan[2] + tab.scan[3];
    const int L = max(max(tab.scan[4], tab.scan[5]), max(tab.scan[6], tab.scan[7]));
    const int G = gridDim.x, pairs = ng * HKV, tiles = (L + 15) >> 4;
    // Warps per task: as many as the grid has for one round of tasks, no more than the longest sequence has tiles.
    int W = 1;
    while (W < 8 && pairs * (2 * W) <= G * kNumConsumerWarps && W < tiles) W *= 2;
    // Few pairs and long sequences: a CTA per chunk of at least 8 tiles, as many chunks as one round of CTAs holds.
    int nch = 1;
    if (W == 8) nch = max(1, min(min(G / pairs, tiles / 8), p.attn_max_chunks));
    const int tpc = (tiles + nch - 1) / nch;  // tiles per chunk
    nch = (tiles + tpc - 1) / tpc;
    tab.plan[0] = ng;
    tab.plan[1] = W;
    tab.plan[2] = nch;
    tab.plan[3] = tpc * 16;
  }
  consumer_sync();
}

// q and k head vectors of the new tokens, where no linear's epilogue has done it: a half-warp per head vector.
__device__ __forceinline__ void attn_prepare_rows(Ctx& c, const OpDesc& op, int T) {
  const int HKV = op.aux0, qpk = op.aux1 / op.aux0, parts = qpk + 2;
  const int total = T * HKV * parts, l16 = c.lane & 15;
#pragma unroll 1
  for (int i0 = (blockIdx.x * kNumConsumerWarps + c.warp) * 2; i0 < total; i0 += gridDim.x * kNumConsumerWarps * 2) {
    const int i = min(i0 + (c.lane >> 4), total - 1);
    const int tok = i / (HKV * parts), e = i % (HKV * parts);
    const __nv_bfloat16* src = reinterpret_cast<const __nv_bfloat16*>(op.in) + (size_t)tok * op.ld_in + (size_t)e * kHeadDim;
    wide_store_head(c, op, __ldcg(reinterpret_cast<const uint4*>(src) + l16), tok, e / parts, e % parts, i0 + (c.lane >> 4) < total, l16);
  }
}

// A group has eight rows: rows 8..15 of the score mma's M side are nothing (shared accumulators in their place would chain
// every mma to the one before).
__device__ __forceinline__ void wide_mma_qk(float (&d)[2], uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1) {
  float x0, x1;
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%10,%10};"
      : "+f"(d[0]), "+f"(d[1]), "=f"(x0), "=f"(x1)
      : "r"(a0), "r"(0u), "r"(a2), "r"(0u), "r"(b0), "r"(b1), "f"(0.f));
}

// Cache rows of a 16-position tile.  Positions at or beyond p1 read row p1 - 1 instead: their probabilities are zero.
__device__ __forceinline__ int wide_page(const Ctx& c, const WideTask& a, int pos) {
  return __ldcg(c.p.kv_indices + a.kvb + (min(pos, a.p1 - 1) >> c.p.page_shift));
}
// this lane's 16-byte column (vector `col` of the head) of the cache row of position `pos`
__device__ __forceinline__ const uint4* wide_row(const Ctx& c, const WideTask& a, const void* cache, int HKV, int pos, int pg, int col) {
  pos = min(pos, a.p1 - 1);
  if (c.p.page_shift < 4) pg = wide_page(c, a, pos);  // (pages of 16 positions or more: one page per tile, looked up ahead)
  const int r = (pg << c.p.page_shift) + (pos & (c.p.page_size - 1));
  return reinterpret_cast<const uint4*>(cache) + ((size_t)r * HKV + a.h) * (kHeadDim / 8) + col;
}
__device__ __forceinline__ void wide_load_k(const Ctx& c, const OpDesc& op, const WideTask& a, int pos0, int pg, uint4 (&kr)[2][4]) {
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const uint4* src = wide_row(c, a, op.k_cache, op.aux0, pos0 + 8 * u + (c.lane >> 2), pg, c.lane & 3);
#pragma unroll
    for (int i = 0; i < 4; ++i) kr[u][i] = __ldcg(src + 4 * i);
  }
}
__device__ __forceinline__ void wide_load_v(const Ctx& c, const OpDesc& op, const WideTask& a, int pos0, int pg, uint4 (&vr)[4][2]) {
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const uint4* src = wide_row(c, a, op.v_cache, op.aux0, pos0 + 2 * (c.lane & 3) + (r & 1) + 8 * (r >> 1), pg, c.lane >> 2);
    vr[r][0] = __ldcg(src);
    vr[r][1] = __ldcg(src + 8);
  }
}
// Two floats as the sum of three bf16 pairs: 24 bits, nothing is lost
__device__ __forceinline__ void split3(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = pack2(a, b);
  a -= bf_lo(hi);
  b -= bf_hi(hi);
  mid = pack2(a, b);
  lo = pack2(a - bf_lo(mid), b - bf_hi(mid));
}

// A task whose output is not finite, once more.  An mma multiplies every row by every V row of its tile: by P = 0 where a
// causal row does not see the position or the tile runs past the end, and by three parts of P of either sign elsewhere, so
// 0 x inf would carry an infinite value of a prompt chunk's last token into the tokens before it.  Here a row takes the
// positions it sees and no others, in scalar fp32: a warp per row, a lane per position for the scores and four dims per
// lane for the sums.  `q0`: the task's q rows, `ld` apart from token to token (read past L1: other CTAs may have written
// them); emit(row, dims 4 lane .. + 3, sums, max, sum of exponentials).  (The check sits on the outputs: 36 layers at 8
// requests 5.83 -> 5.86 ms when it was added; on the accumulators, with the sums redone in place, 5.90.)
template <class Emit>
__device__ __forceinline__ void attend_exact(const KParams& p, const OpDesc& op, const WideTask& a, int W, const __nv_bfloat16* q0, size_t ld, int ldh, Emit emit) {
  const int HKV = op.aux0, qpk = op.aux1 / HKV, rows = a.nt * qpk, lane = threadIdx.x & 31;
  const float sc = 1.4426950408889634f * 0.08838834764831845f;  // log2(e) / sqrt(128)
#pragma unroll 1
  for (int r = (threadIdx.x >> 5) & (W - 1); r < rows; r += W) {
    const int tok = r / qpk, head = r % qpk, last = min(a.L0 + tok, a.p1);
    const volatile uint32_t* q = reinterpret_cast<const volatile uint32_t*>(q0 + (size_t)tok * ld + (size_t)head * ldh);
    float M = -INFINITY, L = 0.f, O[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {  // the maximum, then the sums
#pragma unroll 1
      for (int pos0 = a.p0; pos0 < last; pos0 += 32) {
        const int pos = min(pos0 + lane, last - 1);
        const int slot = (__ldcg(p.kv_indices + a.kvb + (pos >> p.page_shift)) << p.page_shift) + (pos & (p.page_size - 1));
        const uint2* k = reinterpret_cast<const uint2*>(op.k_cache) + ((size_t)slot * HKV + a.h) * (kHeadDim / 4);
        float s = 0.f;
#pragma unroll 1
        for (int i = 0; i < kHeadDim / 4; ++i) {
          const uint32_t qa = q[2 * i], qb = q[2 * i + 1];
          const uint2 kk = __ldcg(k + i);
          s = fmaf(bf_lo(qa), bf_lo(kk.x), s);
          s = fmaf(bf_hi(qa), bf_hi(kk.x), s);
          s = fmaf(bf_lo(qb), bf_lo(kk.y), s);
          s = fmaf(bf_hi(qb), bf_hi(kk.y), s);
        }
        s = pos0 + lane < last ? s * sc : -INFINITY;
        if (pass == 0) {
          M = fmaxf(M, s);
          continue;
        }
        const float pr = exp2f(s - (M == -INFINITY ? 0.f : M));
        L += pr;
#pragma unroll 1
        for (int i = 0; i < min(32, last - pos0); ++i) {
          const int vs = __shfl_sync(0xffffffffu, slot, i);
          const float pi = __shfl_sync(0xffffffffu, pr, i);
          const uint2 v = __ldcg(reinterpret_cast<const uint2*>(op.v_cache) + ((size_t)vs * HKV + a.h) * (kHeadDim / 4) + lane);
          O[0] = fmaf(pi, bf_lo(v.x), O[0]);
          O[1] = fmaf(pi, bf_hi(v.x), O[1]);
          O[2] = fmaf(pi, bf_lo(v.y), O[2]);
          O[3] = fmaf(pi, bf_hi(v.y), O[3]);
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        if (pass == 0) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
        else L += __shfl_xor_sync(0xffffffffu, L, o);
      }
    }
    emit(r, 4 * lane, make_float4(O[0], O[1], O[2], O[3]), M, L);
  }
}
// bar.sync that also tells every thread whether any thread's `pred` holds
__device__ __forceinline__ bool bar_any(int id, int nthr, bool pred) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %3, 0;\n\tbar.red.or.pred q, %1, %2, p;\n\tselp.b32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"(id), "r"(nthr), "r"((uint32_t)pred)
      : "memory");
  return r != 0u;
}

// The tiles ti, ti + W, ... of a task by one warp: (max, sum) of row g and, per tile t of 16 dims, oacc[t] = {dim 8 g + t of rows 2 j and
// 2 j + 1, dim 64 + 8 g + t of the same}.  The first tile's rows are in kr and vr, pgn is the page of the second.  FRESH: K and V of
// the positions from a.fresh on are the two rows at fresh_kv (the new token's, in shared memory), not the cache's.
template <bool FRESH>
__device__ __forceinline__ void attend_tiles(const Ctx& c, const OpDesc& op, const WideTask& a, int W, int ti, int pgn, const uint4 (&qf)[4],
                                             uint4 (&kr)[2][4], uint4 (&vr)[4][2], const uint4* fresh_kv, float& m, float& l, float (&oacc)[8][4]) {
  const int lane = c.lane, g = lane >> 2, j = lane & 3;
  const int qpk = op.aux1 / op.aux0, psh = c.p.page_shift;
  const int ntiles = (a.p1 - a.p0 + 15) >> 4;
  const float sc = 1.4426950408889634f * 0.08838834764831845f;  // log2(e) / sqrt(128)
  m = -INFINITY;
  l = 0.f;
#pragma unroll
  for (int t = 0; t < 8; ++t)
#pragma unroll
    for (int i = 0; i < 4; ++i) oacc[t][i] = 0.f;
  const int last = min(a.L0 + g / qpk, a.p1);  // positions row g sees: it belongs to token g / qpk of the group
#pragma unroll 1
  for (; ti < ntiles; ti += W) {
    const int pos0 = a.p0 + 16 * ti;
    const bool more = ti + W < ntiles;
    if constexpr (FRESH) {
      if (pos0 + 15 >= a.fresh) {  // rows from a.fresh on (and what a position past the end is clamped to) come from shared memory
#pragma unroll
        for (int u = 0; u < 2; ++u)
          if (min(pos0 + 8 * u + g, a.p1 - 1) >= a.fresh)
#pragma unroll
            for (int i = 0; i < 4; ++i) kr[u][i] = fresh_kv[j + 4 * i];
#pragma unroll
        for (int r = 0; r < 4; ++r)
          if (min(pos0 + 2 * j + (r & 1) + 8 * (r >> 1), a.p1 - 1) >= a.fresh) {
            vr[r][0] = fresh_kv[16 + g];
            vr[r][1] = fresh_kv[24 + g];
          }
      }
    }
    float s0[2] = {0.f, 0.f}, s1[2] = {0.f, 0.f}, z0[2] = {0.f, 0.f}, z1[2] = {0.f, 0.f};
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      const uint2 qa = (s & 1) ? make_uint2(qf[s >> 1].z, qf[s >> 1].w) : make_uint2(qf[s >> 1].x, qf[s >> 1].y);
      const uint4 &k0 = kr[0][s >> 1], &k1 = kr[1][s >> 1];
      wide_mma_qk((s & 1) ? z0 : s0, qa.x, qa.y, (s & 1) ? k0.z : k0.x, (s & 1) ? k0.w : k0.y);
      wide_mma_qk((s & 1) ? z1 : s1, qa.x, qa.y, (s & 1) ? k1.z : k1.x, (s & 1) ? k1.w : k1.y);
    }
    if (more) wide_load_k(c, op, a, pos0 + 16 * W, pgn, kr);  // K of the next tile flies during the rest of this one
    // row g, positions pos0 + 2 j + {0, 1} and pos0 + 8 + 2 j + {0, 1}
    float sv[4] = {s0[0] + z0[0], s0[1] + z0[1], s1[0] + z1[0], s1[1] + z1[1]};
    float tmax = -INFINITY;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      sv[i] = pos0 + 2 * j + (i & 1) + 8 * (i >> 1) < last ? sv[i] * sc : -INFINITY;
      tmax = fmaxf(tmax, sv[i]);
    }
    tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, 1));
    tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, 2));
    const float mn = fmaxf(m, tmax);
    const float ms = mn == -INFINITY ? 0.f : mn;  // (a causal row may see nothing of a tile)
    const float alpha = exp2f(m - ms);
    m = mn;
#pragma unroll
    for (int i = 0; i < 4; ++i) sv[i] = exp2f(sv[i] - ms);
    l = l * alpha + ((sv[0] + sv[1]) + (sv[2] + sv[3]));  // this lane's share: the quad adds up at the end
    uint32_t ph[2], pm[2], pl[2];  // as they are, the B operand of O^T = V^T P^T
    split3(sv[0], sv[1], ph[0], pm[0], pl[0]);
    split3(sv[2], sv[3], ph[1], pm[1], pl[1]);
    const float al0 = __shfl_sync(0xffffffffu, alpha, 8 * j), al1 = __shfl_sync(0xffffffffu, alpha, 8 * j + 4);  // rows 2 j, 2 j + 1
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      oacc[t][0] *= al0;
      oacc[t][1] *= al1;
      oacc[t][2] *= al0;
      oacc[t][3] *= al1;
      // element t of the lane's two vectors of four V rows, two rows per register
      uint32_t e[4][2];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int x = 0; x < 2; ++x) e[r][x] = t < 2 ? vr[r][x].x : (t < 4 ? vr[r][x].y : (t < 6 ? vr[r][x].z : vr[r][x].w));
      const uint32_t sel = (t & 1) ? 0x7632u : 0x5410u;
      const uint32_t a0 = prmt(e[0][0], e[1][0], sel), a1 = prmt(e[0][1], e[1][1], sel);
      const uint32_t a2 = prmt(e[2][0], e[3][0], sel), a3 = prmt(e[2][1], e[3][1], sel);
      mma_bf16(oacc[t], a0, a1, a2, a3, ph[0], ph[1]);
      mma_bf16(oacc[t], a0, a1, a2, a3, pm[0], pm[1]);
      mma_bf16(oacc[t], a0, a1, a2, a3, pl[0], pl[1]);
    }
    if (more) {
      wide_load_v(c, op, a, pos0 + 16 * W, pgn, vr);
      if (psh >= 4) pgn = ti + 2 * W < ntiles ? wide_page(c, a, pos0 + 32 * W) : 0;
    }
  }
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);
}

// emit(batch, row, dims d .. d + 3, sums, max, sum of exponentials) for every output of the task
template <class Emit>
__device__ __forceinline__ void attend_combine(const Ctx& c, int W, int gi, int rows, uint8_t* reg, float2* ml, float m, float l, const float (&oacc)[8][4],
                                               Emit emit) {
  const int lane = c.lane, g = lane >> 2, j = lane & 3;
  const int sub = c.warp & (W - 1), gtid = sub * 32 + lane, nthr = W * 32;
  // The warps of the task meet in shared memory, four rows at a time: the upper half leaves its sums in W / 2 slots, the
  // lower half adds its own to them, in place, and all finish the rows from there.
  const uint32_t nbar = (uint32_t)(2 + gi);
  const int H = W >> 1;
  if (j == 0) ml[c.warp * 8 + g] = make_float2(m, l);
  float* slot0 = reinterpret_cast<float*>(reg);
#pragma unroll
  for (int rb = 0; rb < 2; ++rb) {
    if (4 * rb >= rows) break;
    if (rb > 0) asm volatile("bar.sync %0, %1;" ::"r"(nbar), "r"(nthr) : "memory");  // (the slots are free again)
    const bool mine = (j >> 1) == rb;  // this lane holds rows 2 j and 2 j + 1
    float* own = slot0 + (size_t)(sub & (H - 1)) * 4 * kHeadDim + 2 * (j & 1) * kHeadDim + 8 * g;
    if (mine && sub >= H) {
#pragma unroll
      for (int y = 0; y < 2; ++y)
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
          for (int i = 0; i < 8; i += 4)
            *reinterpret_cast<float4*>(own + y * kHeadDim + 64 * x + i) =
                make_float4(oacc[i][2 * x + y], oacc[i + 1][2 * x + y], oacc[i + 2][2 * x + y], oacc[i + 3][2 * x + y]);
    }
    asm volatile("bar.sync %0, %1;" ::"r"(nbar), "r"(nthr) : "memory");
    const float2* mlt = ml + (c.warp - sub) * 8;  // the task's pairs
    if (mine && sub < H) {
#pragma unroll
      for (int y = 0; y < 2; ++y) {
        const float m0 = mlt[sub * 8 + 2 * j + y].x, m1 = mlt[(sub + H) * 8 + 2 * j + y].x;
        const float M = fmaxf(m0, m1), Ms = M == -INFINITY ? 0.f : M;
        const float f0 = exp2f(m0 - Ms), f1 = exp2f(m1 - Ms);
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
          for (int i = 0; i < 8; i += 4) {
            float4* q = reinterpret_cast<float4*>(own + y * kHeadDim + 64 * x + i);
            const float4 o = *q;
            *q = make_float4(fmaf(f1, o.x, f0 * oacc[i][2 * x + y]), fmaf(f1, o.y, f0 * oacc[i + 1][2 * x + y]),
                             fmaf(f1, o.z, f0 * oacc[i + 2][2 * x + y]), fmaf(f1, o.w, f0 * oacc[i + 3][2 * x + y]));
          }
      }
    }
    asm volatile("bar.sync %0, %1;" ::"r"(nbar), "r"(nthr) : "memory");
#pragma unroll 1
    for (int e = gtid; e < 4 * 32; e += nthr) {  // (row of the round, four dims)
      const int r = 4 * rb + (e >> 5), d = (e & 31) * 4;
      if (r >= rows) continue;
      const float2* mlr = mlt + r;
      float M = -INFINITY;
      for (int w = 0; w < W; ++w) M = fmaxf(M, mlr[w * 8].x);
      const float Ms = M == -INFINITY ? 0.f : M;
      float L = 0.f;
      float4 O = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
      for (int w = 0; w < H; ++w) {
        const float2 v0 = mlr[w * 8], v1 = mlr[(w + H) * 8];
        L = fmaf(exp2f(v0.x - Ms), v0.y, L);
        L = fmaf(exp2f(v1.x - Ms), v1.y, L);
        const float f = exp2f(fmaxf(v0.x, v1.x) - Ms);
        const float4 o4 = *reinterpret_cast<const float4*>(slot0 + (size_t)w * 4 * kHeadDim + (e >> 5) * kHeadDim + d);
        O.x = fmaf(f, o4.x, O.x);
        O.y = fmaf(f, o4.y, O.y);
        O.z = fmaf(f, o4.z, O.z);
        O.w = fmaf(f, o4.w, O.w);
      }
      emit(rb, r, d, O, M, L);
    }
  }
}

// One task by W warps.  `loaded`: the first tile's K and V rows are in kr and vr already, but for the rows that this iteration writes.
// (What is only used behind the tiles is worked out there: held in registers across their loop it cost 0.5 to 1.5 % behind 8000
// positions at 33 and more tokens.)
__device__ __forceinline__ void wide_attend(Ctx& c, const OpDesc& op, const WideTask& a, int W, bool loaded,
                                            uint4 (&kr)[2][4], uint4 (&vr)[4][2]) {
  const KParams& p = c.p;
  const int lane = c.lane, g = lane >> 2, j = lane & 3;
  const int HKV = op.aux0, qpk = op.aux1 / HKV, rows = a.nt * qpk;
  const int sub = c.warp & (W - 1), nthr = W * 32;
  const int psh = p.page_shift;
  const int ntiles = (a.p1 - a.p0 + 15) >> 4;
  int ti = sub;
  // Row g of the q rows as A fragments: 8 dims from 32 i + 8 j are k steps 2 i and 2 i + 1; rows past the group's are zero.
  uint4 qf[4];
  {
    const __nv_bfloat16* q0 = reinterpret_cast<const __nv_bfloat16*>(op.out2) + (size_t)(a.t0 + g / qpk) * op.ld_out2 + (size_t)(a.h * qpk + g % qpk) * kHeadDim + 8 * j;
#pragma unroll
    for (int i = 0; i < 4; ++i) qf[i] = g < rows ? __ldcg(reinterpret_cast<const uint4*>(q0 + 32 * i)) : make_uint4(0, 0, 0, 0);
  }
  if (ti < ntiles && (!loaded || a.p0 + 16 * ti + 15 >= a.fresh)) {
    const int pg = psh >= 4 ? wide_page(c, a, a.p0 + 16 * ti) : 0;
    wide_load_k(c, op, a, a.p0 + 16 * ti, pg, kr);
    wide_load_v(c, op, a, a.p0 + 16 * ti, pg, vr);
  }
  int pgn = (psh >= 4 && ti + W < ntiles) ? wide_page(c, a, a.p0 + 16 * (ti + W)) : 0;
  MK_STAMP(c, 1);
  float m, l, oacc[8][4];
  attend_tiles<false>(c, op, a, W, ti, pgn, qf, kr, vr, nullptr, m, l, oacc);
  MK_STAMP(c, 2);
  __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(op.out) + (size_t)a.t0 * op.ld_out + (size_t)a.h * qpk * kHeadDim;
  float* part = p.attn_part + ((size_t)a.t0 * HKV * p.attn_max_chunks * qpk + (size_t)(a.h * p.attn_max_chunks + a.ch) * rows) * (kHeadDim + 2);
  const __nv_bfloat16* q = reinterpret_cast<const __nv_bfloat16*>(op.out2) + (size_t)a.t0 * op.ld_out2 + (size_t)a.h * qpk * kHeadDim;
  auto store = [&](int r, int d, const float4& O, float M, float L) {
    if (a.nch == 1) {
      const float inv = __fdividef(1.0f, L);
      *reinterpret_cast<uint2*>(out + (size_t)(r / qpk) * op.ld_out + (r % qpk) * kHeadDim + d) =
          make_uint2(pack2(O.x * inv, O.y * inv), pack2(O.z * inv, O.w * inv));
    } else {
      *reinterpret_cast<float2*>(part + r * kHeadDim + d) = make_float2(O.x, O.y);
      *reinterpret_cast<float2*>(part + r * kHeadDim + d + 2) = make_float2(O.z, O.w);
      if (d == 0) {
        part[rows * kHeadDim + r] = M;
        part[rows * kHeadDim + rows + r] = L;
      }
    }
  };
  float chk = 0.f;  // stays zero while the outputs are finite
  if (W == 1 && a.nch == 1) {
#pragma unroll
    for (int y = 0; y < 2; ++y) {
      const float lr = __shfl_sync(0xffffffffu, l, 8 * j + 4 * y);
      const int r = 2 * j + y;
      if (r < rows) {
        const float inv = __fdividef(1.0f, lr);
        __nv_bfloat16* dst = out + (size_t)(r / qpk) * op.ld_out + (r % qpk) * kHeadDim + 8 * g;
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          float f[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            f[i] = oacc[i][2 * x + y] * inv;
            chk = fmaf(f[i], 0.f, chk);
          }
          *reinterpret_cast<uint4*>(dst + 64 * x) = pack8(f);
        }
      }
    }
    __syncwarp();
    if (__any_sync(0xffffffffu, chk != 0.f)) attend_exact(p, op, a, W, q, op.ld_out2, kHeadDim, store);
    return;
  }
  const int gi = c.warp / W;
  uint8_t* reg = c.smem + p.x_off + (size_t)gi * W * 1024;          // the group's shared memory, W KB
  float2* ml = reinterpret_cast<float2*>(c.smem + p.x_off + 8192);  // [warps of the CTA][8] (max, sum) pairs
  const uint32_t nbar = (uint32_t)(2 + gi);
  attend_combine(c, W, gi, rows, reg, ml, m, l, oacc, [&](int, int r, int d, const float4& O, float M, float L) {
    chk = fmaf(O.x, 0.f, fmaf(O.y, 0.f, fmaf(O.z, 0.f, fmaf(O.w, 0.f, chk))));
    store(r, d, O, M, L);
  });
  MK_STAMP(c, 3);
  if (bar_any((int)nbar, nthr, chk != 0.f)) {  // (the group's memory is free again)
    attend_exact(p, op, a, W, q, op.ld_out2, kHeadDim, store);
    asm volatile("bar.sync %0, %1;" ::"r"(nbar), "r"(nthr) : "memory");
  }
  if (a.nch == 1) return;
  // several chunks (then W == 8, the whole CTA): the one that arrives last merges them.  The CTA's partial is complete
  // behind the sync above; thread 0's release publishes all of it.
  unsigned* cnt = p.attn_count + (size_t)a.t0 * HKV + a.h;
  volatile int* fl = c.flags();
  if (c.tid == 0) {
    unsigned old;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(cnt) : "memory");
    fl[2] = (old == (unsigned)(a.nch - 1)) ? 1 : 0;
  }
  consumer_sync();
  if (fl[2] != 0) {
    const int stride = rows * (kHeadDim + 2);
    const float* base = part - (size_t)a.ch * stride;
#pragma unroll 1
    for (int e = c.tid; e < rows * 64; e += kNumConsumers) {
      const int r = e >> 6, d = (e & 63) * 2;
      float M = -INFINITY, L = 0.f;
      float2 O = make_float2(0.f, 0.f);
#pragma unroll 1
      for (int c0 = 0; c0 < a.nch; c0 += 8) {
        float2 v[8];
        float mm[8], ll[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const bool ok = c0 + u < a.nch;
          const float* b = base + (size_t)(ok ? c0 + u : c0) * stride;
          v[u] = ok ? __ldcg(reinterpret_cast<const float2*>(b + r * kHeadDim + d)) : make_float2(0.f, 0.f);
          mm[u] = ok ? __ldcg(b + rows * kHeadDim + r) : -INFINITY;
          ll[u] = ok ? __ldcg(b + rows * kHeadDim + rows + r) : 0.f;
        }
        float Mb = M;
#pragma unroll
        for (int u = 0; u < 8; ++u) Mb = fmaxf(Mb, mm[u]);
        const float Ms = Mb == -INFINITY ? 0.f : Mb;
        const float f0 = exp2f(M - Ms);
        O.x *= f0;
        O.y *= f0;
        L *= f0;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const float f = exp2f(mm[u] - Ms);
          O.x = fmaf(f, v[u].x, O.x);
          O.y = fmaf(f, v[u].y, O.y);
          L = fmaf(f, ll[u], L);
        }
        M = Mb;
      }
      const float inv = __fdividef(1.0f, L);
      *reinterpret_cast<uint32_t*>(out + (size_t)(r / qpk) * op.ld_out + (r % qpk) * kHeadDim + d) = pack2(O.x * inv, O.y * inv);
    }
    if (c.tid == 0) *cnt = 0u;
  }
  consumer_sync();
}

__device__ __forceinline__ void op_attention_wide(Ctx& c, const OpDesc& op, int T) {
  const KParams& p = c.p;
  // What does not depend on the QKV linear before the op is done ahead of its barrier: the plan, and the K and V rows of this warp's
  // first tile.  Rows that this iteration writes are loaded again behind the barrier (the others then hit L2).
  // (The arrival comes first: behind the page look-up it held the others up, 3 % of a step of a small model.)
  if (op.flags & F_SYNC_BEFORE) grid_arrive(c);
  const int key = op.aux0 * 256 + op.aux1;
  if (c.attn_iter != key) {
    wide_plan_attention(c, op, T);
    c.attn_iter = key;
  }
  const WideTab& tab = wide_tab(c);
  const int HKV = op.aux0;
  const int W = tab.plan[1], nch = tab.plan[2], CS = tab.plan[3];
  const int ntasks = tab.plan[0] * HKV * nch, per = kNumConsumerWarps / W;
  const int gi = c.warp / W;
  uint4 kr[2][4], vr[4][2];
  bool loaded = false;
#pragma unroll 1
  for (int task = blockIdx.x + gridDim.x * gi, first = 1;; task += gridDim.x * per, first = 0) {
    WideTask a;
    a.p0 = a.p1 = a.fresh = 0;
    bool live = task < ntasks;
    if (live) {
      a.ch = task % nch;
      const int pr = task / nch;
      a.h = pr % HKV;
      const int e = tab.grp[pr / HKV];
      a.t0 = e & 255;
      a.nt = e >> 8;
      a.L0 = tab.pos[a.t0] + 1;
      a.kvb = tab.kvb[a.t0];
      a.fresh = tab.fresh[a.t0];
      const int L = a.L0 + a.nt - 1;
      a.p0 = a.ch * CS;
      a.p1 = min(L, a.p0 + CS);
      a.nch = (L + CS - 1) / CS;
      live = a.p0 < L && a.L0 > 0;  // (uniform within the task's warps)
    }
    if (first) {
      const int pos0 = a.p0 + 16 * (c.warp & (W - 1));
      if (live && pos0 < min(a.p1, a.fresh) && !(p.debug_flags & 2)) {
        const int pg = p.page_shift >= 4 ? wide_page(c, a, pos0) : 0;
        wide_load_k(c, op, a, pos0, pg, kr);
        wide_load_v(c, op, a, pos0, pg, vr);
        loaded = true;
      }
      if (op_barrier(c, op)) return;
      if (p.debug_flags & 2) return;  // measurement aid: the op keeps its barrier and does nothing else
      if (!(op.flags & F_QKV_READY)) {
        attn_prepare_rows(c, op, T);
        grid_sync(c);  // every token's K/V row is in the cache before any is read
        c.dead = c.flags()[3] != 0;
        if (c.dead) return;
      }
      MK_STAMP(c, 0);
    }
    if (task >= ntasks) break;
    if (live) wide_attend(c, op, a, W, first && loaded, kr, vr);
  }
}
