// Shared host/device definitions of the B200 decode megakernel.
//
// The host runtime lowers the recorded operator list into a flat array of
// OpDesc (the "program").  One persistent cooperative kernel walks that array
// once per decode iteration on every SM.
#pragma once
#include <stdint.h>

namespace mk {

// ---- geometry of the weight stream -------------------------------------------------
// A weight tile is 128 output rows x 128 k-elements of bf16 (32 KB): two 2-D TMA boxes
// of 128 rows x 64 k-elements, adjacent in k, each landing 128-byte-swizzled in its half
// of a shared-memory stage.  One mbarrier round trip per 32 KB keeps the producer and
// consumer loops off the critical path.
constexpr int kTileRows = 128;
constexpr int kBoxK = 64;                         // k-elements of one TMA box (128 bytes: the swizzle span)
constexpr int kSubTiles = 2;                      // boxes per stage, adjacent in k
constexpr int kTileK = kBoxK * kSubTiles;         // k-elements per stage
constexpr int kSubBytes = kTileRows * kBoxK * 2;  // 16 KB
constexpr int kStageBytes = kSubBytes * kSubTiles;
constexpr int kNumConsumerWarps = 8;
constexpr int kNumConsumers = kNumConsumerWarps * 32;
// + a warpgroup of service warps: the weight producer, the activation producer (or L2 look-ahead) and, on the wide path, the
// MMA issuer and the norm warp.  The block starts with kLaunchRegs registers a thread; the service warps hand theirs to the
// consumers (their sum is what the block was launched with; an instance that is compiled to fewer is not launched).  The
// instances with a norm warp, up to 32 token rows, leave it 72: with 56 it has two rows in flight instead of four (12 layers of 8B
// width, us per step: 32 requests 1520 and 1421, 8 requests 1249 and 1237).  On the row-owner path the MoE build's issuer would
// spill with 56, beyond 32 token rows the consumers with 216.
constexpr int kNumThreads = kNumConsumers + 128;
constexpr int kLaunchRegs = 168;
__host__ __device__ constexpr int service_regs(int nc) { return nc == 32 ? 56 : 72; }  // (nc: MK_NC of the instance)
__host__ __device__ constexpr int consumer_regs(int nc) { return (kNumThreads * kLaunchRegs - 128 * service_regs(nc)) / kNumConsumers; }
static_assert(consumer_regs(32) == 224 && consumer_regs(8) == 216, "register counts in steps of eight, no more than the block has");
constexpr int kWideRedBytes = 4096;              // scratch of the wide path: reductions and the iteration's token table
constexpr int kHeadDim = 128;
// Widest activation box that the norm is applied to in shared memory: what one warp normalises in the time a weight stage takes
// to arrive (32 requests, 12 layers of 8B width, with a norm op and in the boxes: 1535 and 1484 us per step; 64 rows not built).
constexpr int kNormBoxRows = 32;
// Columns a stand-alone norm stages in shared memory (48 KB).  Wider rows are read twice instead: at 65 tokens and more,
// where a ring stage is 64 KB, two stages would leave no room for rows of more than 46000 columns.
constexpr int kNormStagedCols = 24576;
// Row-owner linear (one or two batched tokens): a CTA owns a contiguous range of 8-row units
// and walks it in chunks of up to 32 rows; a stage holds a chunk's rows for 512 k-elements
// as eight TMA boxes of 64 k-elements (32 KB for a full chunk).
constexpr int kUnitRows = 8;
constexpr int kChunkRows = 32;
constexpr int kRowsStageK = 512;
// Tensor memory: 512 columns of 128 lanes x 4 bytes.  A slot holds a stage's 32 KB of weights.
constexpr int kTmemCols = 512;
constexpr int kSlotCols = 64;
constexpr int kRowsCombineBytes = kNumConsumerWarps * 4 * kHeadDim * 4;  // row-owner attention: four rows of sums of every warp
constexpr int kRowsBoxBytes = kChunkRows * kBoxK * 2;  // row-owner path: boxes of a stage lie 4 KB apart, however many of their 32 rows there are
// Row-owner path: two sets of four accumulators of 16 columns, then slots.
constexpr int kRowsAccCols = 64;
constexpr int kRowsSlots = (kTmemCols - 2 * kRowsAccCols) / kSlotCols;
// Slots of the wide path's weight ring behind two accumulator buffers of x_rows columns: 7 up to 32 token rows, 6 up to 64, 4 beyond.
__host__ __device__ constexpr int wide_slots(int x_rows) { return (kTmemCols - 2 * x_rows) / kSlotCols; }
// mbarriers of a CTA: six groups of kMaxStages (see Ctx in mk_kernel.cu), then flags and the single ones
constexpr int kMaxStages = 8;
constexpr int kFlagsOff = 6 * kMaxStages * 8;
constexpr int kBarBytes = kFlagsOff + 192;
static_assert(wide_slots(16) <= kMaxStages && kRowsSlots <= kMaxStages, "a barrier per slot");

enum OpType : int {
  OP_EMBED = 1,
  OP_RMSNORM = 2,
  OP_LINEAR = 3,
  OP_ATTN = 4,
  OP_SILU_MUL = 5,
  OP_ARGMAX_PARTIAL = 6,
  OP_ARGMAX_REDUCE = 7,
  OP_ALLREDUCE = 8,
  // mixture of experts (one or two batched tokens: every (token, expert slot) pair is a row-owner GEMV)
  OP_MOE_ROUTE = 9,    // router logits [T, experts] -> top-k expert ids and renormalised softmax weights
  OP_MOE_LINEAR = 10,  // out[pair] = W[expert of the pair] * in[token or pair]; n = rows per expert, aux1 = experts
  OP_MOE_COMBINE = 11, // out[t] = sum over the token's slots of weight * in[pair] (+ residual)
};

enum OpFlags : int {
  F_SYNC_BEFORE = 1 << 0,   // grid barrier before the op
  F_CTA0_ONLY = 1 << 1,     // only CTA 0 executes the body
  F_NORM_IN = 1 << 2,       // linear: RMSNorm fused on the input rows (wide path: applied to the activation boxes in shared memory, the row
                            // sums of squares come from the linear before, F_ROW_SUMS: ll_in, ll_in_op of them per token)
  F_RESIDUAL = 1 << 3,      // linear: + residual
  F_SILU_MUL = 1 << 4,      // linear: rows are [4 gate | 4 up] per 8-row unit, epilogue SiLU(gate)*up (MoE gate/up: a chunk is [gate | up] halves, also -> out2)
  F_ARGMAX = 1 << 5,        // linear: per-tile (max, index) of the bf16 logits
  F_QK_NORM = 1 << 6,       // attention
  F_ROPE = 1 << 7,          // attention
  F_ROW_SUMS = 1 << 25,     // wide linear: the epilogue also stores, per token, the sum of squares of every 32 output columns (ll_out, ll_res_op of them per token)
  F_RES_RANK0 = 1 << 9,     // residual only contributed when rank == 0 (row-parallel TP)
  F_QKV_PREP = 1 << 8,      // wide QKV linear: the epilogue applies QK-norm and RoPE, stores q to the attention's scratch rows (out2)
                            // and k / v to the cache (aux0/aux1: kv/q heads, aux2: cos/sin rows, aux3: F_QK_NORM | F_ROPE)
  F_QKV_READY = 1 << 10,    // wide attention: the linear before it has F_QKV_PREP
  F_ROWS = 1 << 11,         // linear: every CTA owns whole output rows (no split over k between CTAs)
  // tensor parallelism: the allreduce behind a row-parallel linear folded into its neighbours
  F_PUSH = 1 << 12,         // linear: the epilogue stores its fp32 sums into every rank's exchange slots instead of `out`
  F_GATHER_IN = 1 << 13,    // linear / rmsnorm: the input rows are the rank-order sum of the latest exchange's slots
  F_GATHER_RES = 1 << 14,   // linear: the residual is the rank-order sum of the latest exchange's slots
  F_MOE_PAIR_IN = 1 << 17,  // MoE linear: the input has one row per (token, slot) pair (the down projection), not one per token
  F_XRANK = 1 << 16,        // argmax reduce: the per-rank (value, index) pairs of a vocabulary-sharded LM head are exchanged and the global best is taken
  // Tagged activations (row-owner path): a producer also stores its bf16 outputs as 8-byte words
  // {two adjacent columns, tag of the producing op in this iteration}; a consumer polls the words
  // it needs instead of waiting at a grid barrier, so data and "ready" arrive in one load.
  F_LL_OUT = 1 << 18,       // linear / attention: the outputs are also stored as tagged words (ll_out)
  F_LL_IN = 1 << 19,        // linear / attention: the input rows are read from tagged words (ll_in, producer op ll_in_op); no barrier
  F_LL_RES = 1 << 20,       // linear: the residual is read from tagged words (ll_res, producer op ll_res_op)
  F_MOE_COMBINE = 1 << 23,  // MoE down linear: a CTA owns output rows for ALL expert slots of a token and adds the slots up itself
                            // (weights amax_val, + res), out: [T, n]; no per-slot output, no separate weighted-sum op
  F_MOE_ROUTE = 1 << 22,    // MoE gate/up linear: the op first routes the tokens itself (res: router logits [T, experts]); every CTA
                            // keeps the expert ids in shared memory for its producer, CTA 0 also stores the runtime's tables
  F_FOLDED = 1 << 24,       // silu_mul behind a MoE gate/up linear with F_SILU_MUL: nothing left to do, no barrier
  F_XRED = 1 << 21,         // linear with F_LL_IN under tensor parallelism: the op first adds up its slice of the latest exchange
                            // over the ranks and stores it as tagged words (ll_in, tagged as its own output), then reads them all
};

enum Numerics : int {
  NUM_MPK = 0,    // fp32 task arithmetic of the reference megakernel, one bf16 rounding per task
  NUM_TORCH = 1,  // bf16 roundings of the reference PyTorch model (no-eps bf16 RMSNorm, ...)
};

enum Mode : int { MODE_OFFLINE = 0, MODE_ONEPASS = 1 };

// The kernel is compiled once per linear-layer path, each instance holding only the code its
// path runs: the whole step executes out of the instruction cache once per layer, and code
// that is merely present (other paths' loops) measurably slowed the batch-1 step down.
enum Path : int {
  PATH_ROWS = 0,  // 1-2 tokens: row-owner linears, resident token rows, L2 look-ahead
  PATH_WIDE = 1,  // 3-128 tokens (and graphs the row-owner path cannot take): stream-K tiles, tcgen05.mma
};

enum Status : int {
  ST_OK = 0,
  ST_TIMEOUT_GRID = 1,
  ST_TIMEOUT_FULL = 2,
  ST_TIMEOUT_EMPTY = 3,
  ST_TIMEOUT_GO = 4,
  ST_TIMEOUT_PEER = 5,
  ST_BAD_TOKEN = 6,
  ST_OUT_OF_PAGES = 7,
  ST_TIMEOUT_RANK = 8,
  ST_TIMEOUT_DATA = 9,
};

struct alignas(16) OpDesc {
  int type;
  int flags;
  // generic shapes
  int n;        // linear: output features; rmsnorm/silu: columns; argmax: vocab
  int k;        // linear: input features
  int ld_in, ld_out, ld_res, ld_out2;  // row pitches in elements
  int nblk, nkt;                       // linear: row tiles, k tiles (F_ROWS: nkt = 512-wide k stages)
  int aux0, aux1, aux2, aux3;          // per-type small ints (see mk_kernel.cu)
  const void* in;
  const void* w;       // linear weight / embedding table / rmsnorm weight
  const void* norm_w;  // fused input norm weight
  const void* res;
  void* out;
  void* out2;
  const void* tmap_w;  // device address of the CUtensorMap of w
  // attention
  const void* tmap_x;     // linear, wide batches: device address of the CUtensorMap of the input rows
  void* k_cache;
  void* v_cache;
  const void* q_norm_w;
  const void* k_norm_w;
  const void* cos;
  const void* sin;
  // argmax partials
  float* amax_val;
  int* amax_idx;
  int amax_n;   // number of partials per token
  int pad_;
  // tagged activations: word (token t, column pair j) of a tensor with row pitch ld sits at [t * (ld / 2) + j]
  const void* ll_in;
  void* ll_out;
  const void* ll_res;
  int ll_in_op, ll_res_op;  // program indices of the ops that produce ll_in / ll_res
};

struct KParams {
  const OpDesc* ops;
  int num_ops;
  int mode;
  int path;  // Path: which instance of the kernel the host launches
  int numerics;
  int rank, world;
  // meta tensors of the operator API (caller-owned)
  int* step;
  long long* tokens;
  long long* input_tokens;
  long long* output_tokens;
  int* num_new_tokens;
  int* prompt_lengths;
  int* qo_indptr;
  int* kv_indptr;
  int* kv_indices;
  int* kv_last_page_len;
  int max_seq_len, max_reqs, max_tokens, max_pages, page_size, total_requests;
  int max_tokens_per_req;  // prompt tokens one request may get per iteration (chunked prefill)
  // A handle may hold two programs over the same state: one planned for iterations of at most
  // max_reqs tokens (decode) and one for the larger iterations that carry prompt chunks.  A launch
  // serves iterations of tok_lo .. tok_hi tokens and hands any other to the host, which launches
  // the other program (ctrl[0] = -2, the prepared token count in sched[5]).
  int tok_lo, tok_hi;
  int page_shift;  // log2(page_size): page sizes are powers of two
  long long eos;
  int vocab_limit;  // embedding rows, to refuse out-of-range token ids
  // runtime-owned state
  int* request_ids;   // [max_reqs]
  int* page_queue;    // ring of free pages [max_pages]
  int* page_scratch;  // [max_pages] copy of the page table while it is rewritten, where it is longer than ...
  int page_entries;   // ... the entries that the weight ring and the x region of shared memory hold
  int* sched;         // [0]=page head [1]=page tail [2]=next request id [3]=iterations done
                      // [4]=outputs of the last iteration not appended yet
                      // [5]=tokens of an iteration that is prepared but was handed to the other program
                      // [6]=exchanges executed by the last launch
                      // [7]=iterations completed by earlier kernels of the current generation call
  unsigned* grid_bar;
  int cluster;            // CTAs per thread-block cluster of the launch (1 = flat grid barrier)
  unsigned bar_epoch0;    // barrier epoch the launch starts at (the counter is preset to match; tests start near the wrap)
  int* ctrl;          // [0] = active tokens of the iteration, -1 = terminate, -2 = hand over to the other program
  int* abort_flag;
  int* status;        // [0]=code [1]=cta [2]=op [3]=iter [4..7]=detail
  unsigned long long* step_times;
  int max_step_times;
  int max_iters;      // 0 = unlimited
  unsigned long long timeout_ns;
  // split-k scratch shared by all linear ops of the wide path
  uint4* partial;         // sums of blocks that several CTAs hold, two slots a CTA (for the CTAs that may hold any: see the host).  Up to
                          // 32 token rows [CTAs][2][x_rows / 2][128 rows] words {sum, tag, sum of the next token, tag}, beyond
                          // [CTAs][2][x_rows / 4][128 rows] float4
  unsigned* piece_flag;   // [CTAs][2][8 warps]: tag of the op whose piece is there (beyond 32 token rows)
  // attention scratch
  float* attn_part;       // [tokens][kv heads][max chunks][qpk*(128+2)]
  unsigned* attn_count;   // [tokens][kv heads]
  int attn_max_chunks;
  uint2* attn_part_ll;    // the same partials as tagged 8-byte words {fp32, tag}, for the merge without a counter (null: not used)
  // tensor-parallel exchange: every rank's exchange region mapped into this GPU's address space
  // (xchg[rank] is the local one).  A region holds slots [2][world][xchg_tokens][xchg_cols] of 8-byte
  // words {fp32 value, sequence number}: a word is valid for exchange number s once its second half
  // equals s, so data and "arrived" flag travel in one store and no fence or separate flag is needed.
  // Exchange s uses the half of the region selected by s & 1 (see xchg_word).
  unsigned char* xchg[8];
  int xchg_tokens, xchg_cols;
  // behind the slots: [world][xchg_tokens][2] words {logit value, number} {vocabulary index, number} for the
  // argmax of a vocabulary-sharded LM head (one buffer: a rank cannot be a whole iteration ahead of a peer)
  long long xchg_amax_word;  // index of that area, in 8-byte words
  unsigned xchg_seq_base;  // exchanges executed by all earlier launches: sequence numbers keep growing (mod 2^32)
  // optional per-op trace of the last iteration: [(op * grid + cta) * 4 + k] globaltimer ns,
  // k = 0 op reached, 1 barrier passed, 2 op done; op == num_ops is the iteration prologue
  unsigned long long* prof;
  int trace_op;     // op whose inner phases are stamped: prof[(num_ops + 1) * grid * 4 + cta * 16 + k]; -1 none
  int debug_flags;  // bit 0: linear tasks of the row-owner path skip the arithmetic (the wide path's MMA issuer does not look
                    // at it: the look cost 0.4 % of a step); bit 1: attention tasks keep their barrier and do nothing else
  int has_attn;        // (wide path) the program holds attention ops: the token table is filled every iteration
  int prefetch_tiles;  // weight tiles per CTA requested into L2 ahead of the ring (0 = off)
  int has_moe;         // the program holds mixture-of-experts ops: the host launches the build of the kernel that has them
  // shared-memory carve-up (bytes from the 1024-aligned base)
  int num_stages;
  int stage_bytes;  // weights (kStageBytes) + on the wide path a stage of the activation boxes' ring
  int x_rows;       // token rows of an activation box (wide path: 16, 32, 64 or 128; row-owner path: 0)
  int sums_off;     // per-(row, token) sums of a run of tiles: [128][sums_stride] floats
  int sums_stride;
  int x_off, x_bytes;
  int red_off;
  int bar_off;
  int desc_off;     // two op descriptors
};

// Exchange sequence arithmetic (shared with the host-side checks).  Exchange k (1-based) of a launch
// that follows `total_before` completed exchanges has number total_before + k, modulo 2^32; number 0 is
// skipped by nobody: a word is "arrived" only when it carries exactly the awaited number, and the
// previous occupants of a slot carry numbers that differ from it by a multiple of 2 up to the region's
// age, so a collision needs 2^32 exchanges between two uses of one slot.
__host__ __device__ inline unsigned xchg_seq(unsigned total_before, unsigned k) { return total_before + k; }
__host__ __device__ inline unsigned xchg_half(unsigned seq) { return seq & 1u; }
__host__ __device__ inline bool xchg_arrived(unsigned word_seq, unsigned seq) { return word_seq == seq; }
// index (in 8-byte words) of (exchange seq, source rank, token row, column) in a region
__host__ __device__ inline size_t xchg_word(unsigned seq, int world, int tokens, int cols, int src, int tok, int col) {
  return (((size_t)xchg_half(seq) * world + src) * tokens + tok) * cols + col;
}

// Tag of the words op `op` stores in iteration `iter` (1-based) of a launch.  The host clears the word
// buffers before every launch, and tags grow with (iteration, op), so a buffer never holds the awaited
// tag before its producer in this iteration has stored it.
__host__ __device__ inline unsigned ll_tag(int iter, int num_ops, int op) {
  return (unsigned)(iter - 1) * (unsigned)num_ops + (unsigned)op + 1u;
}

// Weight tiles of a linear op are dealt to `grid` CTAs as contiguous ranges
// [c*total/grid, (c+1)*total/grid); tile_owner is the inverse.  32-bit arithmetic: the
// host refuses ops with total * (grid + 1) >= 2^32 tiles.
__host__ __device__ inline unsigned tile_begin(unsigned c, unsigned total, unsigned grid) {
  return c * total / grid;
}
__host__ __device__ inline int tile_owner(unsigned tile, unsigned total, unsigned grid) {
  return (int)(((tile + 1u) * grid - 1u) / total);
}
// CTAs that share a wide linear of nblk row blocks x nkt k tiles: all of them, a tile each where there are fewer tiles.
// (A CTA per whole block, without an exchange of sums, from 33 tokens and up to nine tiles a block, was taken back: an mma
// chain truncates what it adds up, and over 8 tiles it misrounds 0.059 % of the outputs; split over CTAs and added in fp32
// 0.010 %.  It gave 6 layers at 64 requests 517 instead of 538 us at 512 hidden, 621 to 628 instead of 637 and, with eight
// kv heads, 743 instead of 726 at 1024; with the tiles of a whole block added one by one in registers 540, 646 and 768.)
__host__ __device__ inline int wide_ctas(int grid, int nblk, int nkt) {
  const unsigned total = (unsigned)nblk * (unsigned)nkt;
  return total < (unsigned)grid ? (int)total : grid;
}

// Whether the CTAs of a row block share its finish (see mk_wide.cuh); x_rows: token rows of a box, T: tokens there are.  It pays
// where no CTA has two groups of tokens to finish in turn: a half's tokens make T / 8 groups up to 32 token rows and T / 16 beyond, and
// a block has ctas / nblk CTAs.  So the line follows the tokens; beyond 64 one CTA takes the block in two rounds, and three
// groups in turn still pay.  Where the CTAs come out even, none is in two blocks, and half as many do beyond 32 rows (74 blocks of 512
// columns: 48 tokens 9.2 and 8.7, 128 13.9 and 12.6; but 24 tokens 7.4 and 8.0).  Linears in a row (barrier each), us by one CTA and
// shared, 48 blocks (6144 rows) of 1024 columns: 24 tokens 8.1 and 7.6, 32 8.3 and 9.5; 48 9.7 and 9.5, 64 10.4 and 11.8; 80 13.9 and
// 13.6; 64 blocks: 24 tokens 8.2 and 9.4, 48 10.1 and 11.8, 80 14.2 and 14.6; 32 blocks: 32 tokens 7.9 and 7.3, 64 9.8 and 9.3, 128
// 15.0 and 14.6.
// Head vectors and the argmax take longer to finish than to fetch: shared up to half as many blocks as CTAs.  12 layers of 8B
// width, 64 requests, QKV (48 blocks) by one CTA and shared 1549 and 1537 us per step; four of 1024, LM head (64 blocks), 17 and 48
// requests 207.5 and 205.5, 238.3 and 234.8.
// Up to 16 token rows shares are of two tokens, and the line lies between QKV of 8B width, which is finished a head vector at a
// time, and its O and down: 16 requests without any of them, with O and down and with all three 1237, 1221 and 1239 us per step.  12 layers
// of 2048 hidden, 4 and 16 requests without any shares 674 and 708, now 652 and 682; four of 1024 185 and 207, now 172 and 200; six of
// 512, 16 requests 247 and 234.
__host__ __device__ inline bool wide_shares(const OpDesc& op, int ctas, int x_rows, int T) {
  int line = x_rows <= 16 ? 4 : 2;
  if (x_rows > 16 && !(op.flags & (F_QKV_PREP | F_ARGMAX)))
    line = x_rows <= 32 ? (T <= 16 ? 2 : (T + 7) / 8) : (ctas % op.nblk == 0 ? 2 : (T > 48 && T <= 64 ? 4 : 3));
  return line * op.nblk <= ctas;
}

static_assert(sizeof(OpDesc) % 16 == 0 && sizeof(OpDesc) <= 256, "OpDesc is copied to shared memory in 16-byte pieces");

}  // namespace mk
