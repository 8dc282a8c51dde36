// BlockRank attention forward on the sm_100a tensor cores (tcgen05 + TMEM), fed by TMA.
//
// Persistent, warp-specialised kernel: one CTA per SM; the CTAs claim work items from a global
// counter.  Two independent "chains" run in every CTA.  A chain owns one 128-row tile at a time
// (128/G consecutive query tokens x the G query heads that share a KV head, so one K/V tile
// serves the whole GQA group and a Q tile is one 3-D TMA box of the [B,S,N,D] tensor), a
// 256-column half of tensor memory (S 128 columns, O 128 columns), a Q buffer, four softmax
// warps, four output warps and its own MMA-issuing warp.  Chains are fed with "jobs" (one row tile against a list
// of 64-key slots) through per-chain record rings and never wait for one another, so one
// chain's MMAs run while the other chain's softmax threads work.
//
// Only live keys are visited:
//   block 0            : own keys, causal
//   document block     : the prefix block's keys, then own keys, causal
//   query (last) block : every slot of the earlier blocks, then own keys, causal
//
// Two kinds of work item:
//   * resident block  (blocks 0 .. M-2 whose prefix + own keys fit the five 64-key slots of
//     shared memory): the block's K/V is loaded ONCE, its row tiles are dealt to the two chains
//     largest first, and every slot is handed back as soon as the remaining (smaller) row tiles
//     of both chains no longer need it, so the next block's loads overlap the tail of this one.
//   * streamed pair   (the query block, cut into chunks of about 1024 context keys that leave
//     un-normalised partials (O, max, sum) merged by attn_combine_kernel; also any block too
//     long to be resident): the two chains take the two row tiles of a pair and walk the same
//     128-key tiles through a two-deep ring.
//
// Roles (640 threads; 61,440 registers at launch, moved to the softmax warps by setmaxnreg):
//   warps 0-3 / 4-7    softmax of chain 0 / 1 (thread = row = TMEM lane); they leave (max, sum) of each finished row
//   warps 8-11 / 12-15 output of chain 0 / 1: O out of tensor memory, normalised, stored, while the softmax warps are at
//                      the next row tile.  (With the softmax warps storing O themselves a row tile cost them 3-5 k cycles
//                      more: 4 prompts of 100 documents 509 us, with these warps 479; one prompt of 5 documents 29.4 and 20.5.)
//   warp 16            TMA producer: claims and decodes items, publishes jobs, loads K/V
//   warps 17 / 18      MMA issuer of chain 0 / 1: S = Q K^T (both operands K-major, 128B swizzle)
//                      and O += P V (P read from tensor memory, V as the MN-major B operand); it also
//                      requests its chain's Q tiles by TMA (it knows when the Q buffer is free)
//   warp 19            zeros in the output's padding slots
// Softmax is base-2, online, with a lazy rescale (O is only touched when the running max grows
// by more than 2^8).  P (bf16, two keys per 32-bit column) overwrites the first half of the S
// tile it was computed from.
//
// Two forms of P (kFine).  Rounded to bf16 it is what head_dim 128 with four heads per KV head has always had here, and the
// reference too.  Every other shape that BRK_ALGO_AUTO brings here has the CUDA-core kernel as its other route, which keeps P
// in fp32; there P goes in as two bf16 parts, P = hi + lo, one product each, and fills the whole S tile ([hi | lo] per 64-key
// slot): what is dropped is below 2^-17 of a probability.  Error of the output against 64 bits (2 heads per KV head, head_dim
// 64, 20 documents of 120..160 tokens): 1.6462e-3 like the CUDA-core kernel, which is the rounding of the output alone; P in
// bf16 2.17e-3.  4 prompts of 20 such documents: 8 heads on 8 58.8 us (P in bf16 53.9, CUDA cores 1,023), 8 heads on one
// 52.6 us (44.0, 901).
//
// What bounds it: the serial steps of a chain, each a few hundred instructions of a few warps, so whatever slows instructions
// slows all of them.  The SM's instruction cache holds 32 KB (straight code runs at one instruction per cycle up to there and
// at a third of that beyond); with several call sites for what a role does the kernel had 117 KB and missed in 6.6 % of
// 62,200 requests per SM (2 prompts of 100 documents), with one site and rolled loops 82 KB and 3.5 % of 56,200.  That, the waits
// and Q tiles prefetched into L2 when their job is published: 4 prompts of 100 documents 476 -> 460 us, of 20 on the padded grid
// 115.5 -> 110.9, one prompt of 100 with raw logits 151.7 -> 146.5, one of 500 documents of 32..256 tokens 579 -> 573 (whole calls).
//
// Shared memory 227 KB: Q 2x32 KB, K pool 80 KB, V pool 80 KB, barriers, job records, row statistics.
// No cluster multicast anywhere.  Every mbarrier wait is bounded (ptx::BoundedWaits); on expiry the thread leaves a code for the
// caller's status word, tries once in every later wait and runs to the normal exit.
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "attn_combine.cuh"
#include "brk_common.cuh"
#include "tc_ptx.cuh"

namespace brk {

// ---- host: tensor maps -----------------------------------------------------------------
EncodeTiledFn get_encode_tiled() {
  static std::atomic<EncodeTiledFn> fn{nullptr};
  if (EncodeTiledFn f = fn.load(std::memory_order_acquire)) return f;
  void* p = nullptr;
  cudaDriverEntryPointQueryResult qres;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) != cudaSuccess ||
      qres != cudaDriverEntryPointSuccess || p == nullptr)
    return nullptr;
  fn.store(reinterpret_cast<EncodeTiledFn>(p), std::memory_order_release);
  return reinterpret_cast<EncodeTiledFn>(p);
}

static int make_tmap(CUtensorMap* out, CUtensorMapDataType type, int bytes, const void* ptr, int D, int heads, int S, int B,
                     int64_t stride_h, int64_t stride_s, int64_t stride_b, int box_h, int box_s) {
  EncodeTiledFn enc = get_encode_tiled();
  BRK_REQUIRE(enc != nullptr, BRK_E_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  if (B == 1) stride_b = (int64_t)S * stride_s;  // a size-1 dim may carry any stride
  cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)heads, (cuuint64_t)S, (cuuint64_t)B};
  cuuint64_t strides[3] = {(cuuint64_t)stride_h * bytes, (cuuint64_t)stride_s * bytes, (cuuint64_t)stride_b * bytes};
  cuuint32_t box[4] = {(cuuint32_t)(128 / bytes), (cuuint32_t)box_h, (cuuint32_t)box_s, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  auto encode = [&] {
    return enc(out, type, 4, const_cast<void*>(ptr), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  };
  CUresult r = encode();
  if (r == CUDA_ERROR_INVALID_CONTEXT || r == CUDA_ERROR_NOT_INITIALIZED) {
    // A thread that has made no runtime call yet (autograd's, with its memory served from the allocator's cache) has no
    // context bound; selecting its device binds it.
    int dev = 0;
    BRK_CUDA(cudaGetDevice(&dev));
    BRK_CUDA(cudaSetDevice(dev));
    r = encode();
  }
  BRK_REQUIRE(r == CUDA_SUCCESS, BRK_E_CUDA,
              "cuTensorMapEncodeTiled failed (%d): dims {%d,%d,%d,%d} strides {%lld,%lld,%lld} box {%d,%d,%d,1}", (int)r,
              D, heads, S, B, (long long)stride_h, (long long)stride_s, (long long)stride_b, 128 / bytes, box_h,
              box_s);
  return BRK_OK;
}

int make_tmap_bf16(CUtensorMap* out, const void* ptr, int D, int heads, int S, int B, int64_t stride_h, int64_t stride_s,
                   int64_t stride_b, int box_h, int box_s) {
  return make_tmap(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, ptr, D, heads, S, B, stride_h, stride_s, stride_b, box_h, box_s);
}
int make_tmap_f32(CUtensorMap* out, const void* ptr, int D, int heads, int S, int B, int64_t stride_h, int64_t stride_s,
                  int64_t stride_b, int box_h, int box_s) {
  return make_tmap(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, ptr, D, heads, S, B, stride_h, stride_s, stride_b, box_h, box_s);
}

namespace {

constexpr int BM = 128;  // query rows (token, head) per row tile
constexpr int BN = 64;   // keys per slot (one TMA box)
constexpr int BT = 128;  // keys per MMA tile (two slots)
constexpr int kSlots = 5;        // 64-key K/V slots in shared memory
constexpr int kMaxGroup = 4;  // consecutive blocks of one (prompt, KV head) per work item, at most
constexpr int kThreads = 640;
constexpr uint32_t kSlotHalf = BN * 128;         // K (or V) of one slot, one 64-wide chunk of head_dim
constexpr uint32_t kPoolHalf = kSlots * kSlotHalf;  // all slots of one chunk, contiguous: key k at k * 128 B
constexpr int kJobRing = 4;                      // published jobs in flight per chain
// Shared-memory layout for head_dim HD (64 or 128): tiles are stored as HD / 64 chunks of 128-byte rows.
template <int HD>
struct Geo {
  static constexpr uint32_t kChunks = HD / 64;
  static constexpr uint32_t kQBytes = kChunks * BM * 128;  // one Q tile
  static constexpr uint32_t kSlotBytes = 2 * kChunks * kSlotHalf;  // K + V of one slot
  static constexpr uint32_t kOffQ = 0;
  static constexpr uint32_t kOffK = kOffQ + 2 * kQBytes;
  static constexpr uint32_t kOffV = kOffK + kChunks * kPoolHalf;
  static constexpr uint32_t kOffBar = kOffV + kChunks * kPoolHalf;
  static constexpr uint32_t kOffJobs = kOffBar + 512;     // 2 x kJobRing records of 16 ints
  static constexpr uint32_t kOffStat = kOffJobs + 2 * kJobRing * 64;  // (max, sum) of each row of a chain's finished tile
  static constexpr uint32_t kSmemBytes = kOffStat + 2 * BM * 8;
  static_assert(kSmemBytes <= 232448, "shared memory per CTA");
};
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kChainCols = 256;  // per chain: S [0,128) (P over its first 64 columns), then O [128,256)
constexpr uint32_t kColO = 128;
constexpr float kLazy = 8.f;
constexpr int kWaitBudget = 1 << 18;
constexpr int kTileFixedCost = 136;  // cost of a row tile beyond its keys (output drain), in keys

enum {
  kQFull = 0,    // +chain  TMA -> MMA: Q tile landed
  kQFree = 2,    // +chain  MMA -> TMA: every QK^T of the job has read Q
  kSFull = 4,    // +chain  MMA -> softmax: S tile complete
  kPFull = 6,    // +chain  softmax -> MMA: P written to tensor memory, S consumed (4 warp arrivals)
  kPVDone = 8,   // +chain  MMA -> softmax: P V of a tile complete
  kOFree = 10,   // +chain  output -> MMA, softmax: O read out of TMEM, row statistics read (4 warp arrivals)
  kKVFull = 12,              // +slot  TMA -> MMA warps: K and V of the slot landed.  Streamed tiles (slots 2i, 2i + 1):
                             //        K on the first slot's barrier, V on the second's, because K can be handed back when its
                             //        Q K^T is done, a softmax pass before V
  kKVFree = kKVFull + kSlots,  // +slot  both MMA warps -> TMA: no MMA still reads the slot (2 arrivals)
  kJobFull = kKVFree + kSlots,            // +chain*kJobRing+i  TMA warp -> MMA warp, softmax warps: record written
  kJobFree = kJobFull + 2 * kJobRing,     // +chain*kJobRing+i  MMA, 4 softmax, 4 output warps -> TMA warp (9 arrivals)
  kOFull = kJobFree + 2 * kJobRing,       // +chain  MMA -> output: the job's last P V complete
  kStat = kOFull + 2,                     // +chain  softmax -> output: row statistics written (4 warp arrivals)
  kNumBars = kStat + 2
};
static_assert(kNumBars * 8 + 8 <= 512, "barrier area");  // + the TMEM base address

// Code for the status word of warp `warp`'s wait on barrier i.
__device__ __forceinline__ int wait_code(int i, int warp) {
  const int x = i & 1;  // (the chain, of the barriers that come in pairs)
  if (i < kQFree) return 20 + x;
  if (i < kSFull) return 28 + x;
  if (i < kPFull) return 30 + x;
  if (i < kPVDone) return 24 + x;
  if (i < kOFree) return 32 + x;
  if (i < kKVFull) return (warp < 8 ? 36 : 26) + x;
  if (i < kKVFree) return 22 + (warp - 17);
  if (i < kJobFull) return 12;
  if (i < kJobFree) return 40 + (i - kJobFull) / kJobRing;
  if (i < kOFull) return 14 + (i - kJobFree) / kJobRing;
  return (i < kStat ? 34 : 38) + x;
}

// Division by a run-time constant with a host-computed reciprocal (round-up method, exact for every
// 32-bit numerator): q = umulhi(n, mul); n / d = (((n - q) >> 1) + q) >> shift.
struct FastDiv {
  uint32_t d, mul, shift;
};
inline FastDiv make_fastdiv(uint32_t d) {
  FastDiv f;
  f.d = d; f.mul = 0; f.shift = 0;
  if (d <= 1) return f;
  uint32_t s = 0;
  while ((1u << s) < d) ++s;  // ceil(log2 d)
  f.mul = (uint32_t)((((uint64_t)1 << 32) * (((uint64_t)1 << s) - d)) / d + 1);
  f.shift = s - 1;
  return f;
}
__device__ __forceinline__ uint32_t fdiv(uint32_t n, const FastDiv& f) {
  if (f.d <= 1) return n;
  const uint32_t q = __umulhi(n, f.mul);
  return (((n - q) >> 1) + q) >> f.shift;
}

struct TcArgs {
  View o;
  float* lse;
  const int32_t* blk_start;
  const int32_t* blk_len;
  int32_t* status;
  int* hdr;         // workspace header: [0] work counter, [1] non-zero if the block spans are malformed
  int B, N, Nk, S, M;
  int G, g_shift;   // query heads per KV head, log2
  float scale_log2;
  int n_split;      // key chunks of the query block's context (1 = no split)
  int lq_max;       // rows per (prompt, head) in the partial buffers (bound on the query block's length)
  int pairs_q;      // row-tile pairs of the query block (covers lq_max)
  int group;        // consecutive blocks 0 .. M-2 of one (prompt, KV head) per work item (their prefix stays resident)
  int n_groups;     // such groups per (prompt, KV head)
  int o_align32;    // output rows are 32-byte aligned (enables 32-byte stores)
  int sec1, total_items;
  FastDiv div_sec1, div_nbg, div_nk;  // by nbg*n_split, nbg, Nk
  int max_block_len, max_query_len;
  int one_wave;       // every CTA has one item: no counter, and the kernel checks the spans itself (no prologue kernel)
  int* work_counter;  // next unclaimed index of the work list (zeroed before the launch)
  float* part_o;    // [B, N, lq_max, n_split, 128] un-normalised partial outputs
  float2* part_ml;  // [B, N, lq_max, n_split] (running max in log2 units, sum)
  const int4* win;    // [B, win_pitch] live 64-key windows of the query block's context, for prompts with padding inside it
  const int* n_live;  // [B] how many, -1: no padding, every window is live (both null in a one-wave call)
  int win_pitch;
};

// Is span j of the (B, M) arrays inside [0, S), no longer than allowed, and behind its predecessor?
__device__ __forceinline__ bool span_ok(const int32_t* blk_start, const int32_t* blk_len, int j, int M, int S, int max_block_len,
                                        int max_query_len) {
  const int m = j % M, s = blk_start[j], l = blk_len[j];
  bool ok = s >= 0 && l >= 0 && l <= max_block_len && s <= S - l;
  if (ok && m > 0) ok = blk_start[j - 1] >= 0 && blk_len[j - 1] >= 0 && blk_start[j - 1] <= s - blk_len[j - 1];
  if (ok && m == M - 1 && max_query_len > 0) ok = l <= max_query_len;
  return ok;
}

// One row tile against a list of 64-key slots: what a chain works on.
constexpr int kFSplit = 1, kFCtxCheck = 2, kFStop = 4, kFDoc = 8, kFFirst = 16, kFKeep = 32, kFWindows = 64;
struct Job {
  int b, g, m, chunk;
  int start, len;        // span of block m
  int t0;                // first token of the row tile
  int n;                 // key slots visible to this row tile (0: nothing to compute, only slots to hand back)
  int ctx_lo, ctx_hi;    // context key range (token slots of the prompt)
  int n_ctx, j0;         // context slots of the block, first slot of this job's list
  int own_n;             // own keys covered by the slot list
  int flags;
  int tile0;             // streamed: ring position (0/1) of the job's first 128-key tile
  int aux;               // streamed: tiles of the item; resident: rel_lo | rel_hi << 8 (slots handed back after the job)
};

// slot j of the job's list -> first key (token slot of the prompt), number of keys, whether it lies in the own block
__device__ __forceinline__ int tile_lo(const Job& it, int j, int& nk, bool& own, int& own_off) {
  const int jg = j + it.j0;
  own = jg >= it.n_ctx;
  if (!own) {
    const int lo = it.ctx_lo + jg * BN;
    nk = min(BN, it.ctx_hi - lo);
    own_off = 0;
    return lo;
  }
  own_off = (jg - it.n_ctx) * BN;
  nk = min(BN, it.own_n - own_off);
  return it.start + own_off;
}

__device__ __forceinline__ void write_record(int* rec, const Job& it) {
  reinterpret_cast<int4*>(rec)[0] = make_int4(it.b, it.g, it.m, it.chunk);
  reinterpret_cast<int4*>(rec)[1] = make_int4(it.start, it.len, it.t0, it.n);
  reinterpret_cast<int4*>(rec)[2] = make_int4(it.ctx_lo, it.ctx_hi, it.n_ctx, it.j0);
  reinterpret_cast<int4*>(rec)[3] = make_int4(it.own_n, it.flags, it.tile0, it.aux);
}
__device__ __forceinline__ Job read_record(const int* rec) {
  const int4 r0 = reinterpret_cast<const int4*>(rec)[0], r1 = reinterpret_cast<const int4*>(rec)[1];
  const int4 r2 = reinterpret_cast<const int4*>(rec)[2], r3 = reinterpret_cast<const int4*>(rec)[3];
  Job it;
  it.b = r0.x; it.g = r0.y; it.m = r0.z; it.chunk = r0.w;
  it.start = r1.x; it.len = r1.y; it.t0 = r1.z; it.n = r1.w;
  it.ctx_lo = r2.x; it.ctx_hi = r2.y; it.n_ctx = r2.z; it.j0 = r2.w;
  it.own_n = r3.x; it.flags = r3.y; it.tile0 = r3.z; it.aux = r3.w;
  return it;
}

// slot -> is it inside some block?  (blk_start is non-decreasing)
__device__ __forceinline__ bool slot_valid(const int32_t* bs, const int32_t* bl, int M, int s) {
  int lo = 0, hi = M;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (bs[mid] <= s) lo = mid + 1; else hi = mid;
  }
  const int m = lo - 1;
  return m >= 0 && s < bs[m] + bl[m];
}

// A claimed work item before decoding: the spans it needs are fetched one item ahead of their use.
//   kind 0: streamed pair p, key chunk `chunk`, of the query block (m = M-1)
//   kind 1: blocks [m, m + cnt) of (b, g); lane i of the warp holds the span of block m + i
struct ItemRaw {
  int kind, p, chunk, b, g, m, cnt;
  int start, len;      // span of block m + lane (kind 1) or of the query block (kind 0)
  int s0, l0;          // span of block 0 (the prefix)
  int s2, l2;          // span of block M-2 (end of the query block's context)
  int live;            // kind 0: live windows of the context, -1: no list
};

// Work list: streamed pairs of the query block first (the longest items), then the groups of blocks 0 .. M-2.
__device__ __forceinline__ ItemRaw load_item(const TcArgs& a, int idx, int lane) {
  ItemRaw r;
  if (idx >= a.total_items) idx = a.total_items - 1;  // prefetch past the end: harmless reload
  const int nbg = a.B * a.Nk;
  int bg;
  if (idx < a.sec1) {
    r.kind = 0;
    r.p = (int)fdiv((uint32_t)idx, a.div_sec1);
    const int q = idx - r.p * (nbg * a.n_split);
    r.chunk = (int)fdiv((uint32_t)q, a.div_nbg);
    bg = q - r.chunk * nbg;
    r.m = a.M - 1;
    r.cnt = 1;
  } else {
    r.kind = 1;
    const int i2 = idx - a.sec1;
    const int grp = (int)fdiv((uint32_t)i2, a.div_nbg);
    bg = i2 - grp * nbg;
    r.m = grp * a.group;
    r.cnt = min(a.group, a.M - 1 - r.m);
    r.p = r.chunk = 0;
  }
  r.b = (int)fdiv((uint32_t)bg, a.div_nk);
  r.g = bg - r.b * a.Nk;
  const int32_t* bs = a.blk_start + (size_t)r.b * a.M;
  const int32_t* bl = a.blk_len + (size_t)r.b * a.M;
  const int m2 = a.M >= 2 ? a.M - 2 : 0;
  const int mm = min(r.m + (r.kind ? lane : 0), a.M - 1);
  r.start = bs[mm];
  r.len = bl[mm];
  r.s0 = bs[0];
  r.l0 = bl[0];
  r.s2 = bs[m2];
  r.l2 = bl[m2];
  r.live = r.kind == 0 && a.n_live ? a.n_live[r.b] : -1;
  return r;
}

// A streamed pair: the two row tiles [2p, 2p+1] of block m against the block's slot list (or one key chunk of it).
struct Pair {
  Job job;         // fields common to both chains
  int t0_0, t0_1;  // first token of each chain's row tile
  int n_0, n_1;    // slots visible to each chain (a prefix of the item's slot list)
  int n_slots;     // slots of the item
  bool valid;
};

__device__ __forceinline__ Pair decode_pair(const TcArgs& a, int b, int g, int m, int chunk, int p, int start, int len,
                                            int s0, int l0, int s2, int l2, int live) {
  Pair pr;
  Job& it = pr.job;
  const int TOK = BM >> a.g_shift;
  it.b = b; it.g = g; it.m = m; it.chunk = chunk;
  it.start = start;
  it.len = len;
  pr.t0_0 = 2 * p * TOK;
  pr.t0_1 = pr.t0_0 + TOK;
  pr.valid = pr.t0_0 < len;
  const bool split = m == a.M - 1 && a.n_split > 1;
  it.flags = split ? kFSplit : 0;
  it.ctx_lo = it.ctx_hi = 0;
  it.n_ctx = it.j0 = it.own_n = 0;
  it.t0 = it.n = it.tile0 = it.aux = 0;
  pr.n_0 = pr.n_1 = pr.n_slots = 0;
  if (!pr.valid) return pr;
  if (m > 0) {
    it.ctx_lo = s0;
    it.ctx_hi = (m < a.M - 1) ? s0 + l0 : s2 + l2;
  }
  const bool on1 = pr.t0_1 < len;
  it.own_n = min(len, (on1 ? pr.t0_1 : pr.t0_0) + TOK);
  it.n_ctx = (it.ctx_hi - it.ctx_lo + BN - 1) / BN;
  if (live >= 0) {  // padding inside the context: its windows come from the list
    it.n_ctx = live;
    it.ctx_hi = it.ctx_lo + live * BN;  // (whole windows; their bits say which keys exist)
    it.flags |= kFWindows | kFCtxCheck;
  }
  const int own_slots = (it.own_n + BN - 1) / BN;
  int j1 = it.n_ctx + own_slots;
  if (split) {
    const int per = (it.n_ctx + a.n_split - 1) / a.n_split;
    it.j0 = min(it.n_ctx, chunk * per);
    if (chunk != a.n_split - 1) j1 = min(it.n_ctx, it.j0 + per);
  }
  pr.n_slots = j1 - it.j0;
  if (pr.n_slots <= 0) {  // a chunk without slots: nothing to do (its partial stays neutral)
    pr.valid = false;
    pr.n_slots = 0;
    return pr;
  }
  // own slots visible to chain x: those starting at or before its last token
  {
    const int own_x = min(own_slots, (min(len, pr.t0_0 + TOK) + BN - 1) / BN);
    pr.n_0 = max(0, min(j1, it.n_ctx + own_x) - it.j0);
  }
  if (on1) {
    const int own_x = min(own_slots, (min(len, pr.t0_1 + TOK) + BN - 1) / BN);
    pr.n_1 = max(0, min(j1, it.n_ctx + own_x) - it.j0);
  }
  return pr;
}

// chain of the i-th largest row tile of a resident block when there are too many tiles to try every split
// (tiles are dealt 0,1,1,0,0,1,1,0,...)
__device__ __forceinline__ int deal_chain(int i) { return ((i & 3) == 0 || (i & 3) == 3) ? 0 : 1; }

// bf16 pair of what bf16 rounding took off x and y; `hi` is their rounded pair (x in the low half)
__device__ __forceinline__ uint32_t low_part(uint32_t hi, float x, float y) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(x - __uint_as_float(hi << 16), y - __uint_as_float(hi & 0xffff0000u));
  return *reinterpret_cast<const uint32_t*>(&v);
}

template <int HD, bool kFine>
__global__ void __launch_bounds__(kThreads, 1)
attn_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
               const __grid_constant__ CUtensorMap tmV, const TcArgs a) {
  using L = Geo<HD>;
  constexpr uint32_t kOffQ = L::kOffQ, kOffK = L::kOffK, kOffV = L::kOffV, kOffBar = L::kOffBar, kOffJobs = L::kOffJobs,
                     kOffStat = L::kOffStat;
  constexpr uint32_t kQBytes = L::kQBytes, kSlotBytes = L::kSlotBytes;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int G = a.G;

  // ---- shared memory carve-up, barriers, TMEM ---------------------------------------------------
  uint8_t* const smem = smem_raw;  // (no static shared memory: the array starts at offset 1024 of the window or a multiple)
  const uint32_t sbase = ptx::smem_u32(smem_raw);
  const uint32_t sBar = sbase + kOffBar;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kOffBar + kNumBars * 8);
  auto bar = [&](int i) { return sBar + (uint32_t)i * 8u; };

  if (tid == 0) {
    for (int i = 0; i < kNumBars; ++i) {
      uint32_t cnt = 1u;
      if ((i >= kPFull && i < kPFull + 2) || (i >= kOFree && i < kOFree + 2) || i >= kStat) cnt = 4u;  // one per warp
      if (i >= kKVFree && i < kKVFree + kSlots) cnt = 2u;                                 // one per MMA warp
      if (i >= kJobFree && i < kOFull) cnt = 9u;                                          // MMA, softmax, output warps
      ptx::mbar_init(bar(i), cnt);
    }
    ptx::fence_barrier_init();
    ptx::prefetch_tmap(&tmQ);
    ptx::prefetch_tmap(&tmK);
    ptx::prefetch_tmap(&tmV);
  }
  __syncwarp();
  if (warp == 0) {
    ptx::tmem_alloc(ptx::smem_u32(tmem_slot), kTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  ptx::grid_dependency_wait();  // (the set-up above runs beside the prologue kernel)
  bool malformed;
  if (a.one_wave) {
    bool bad = false;
    for (int j = tid; j < a.B * a.M; j += kThreads)
      bad |= !span_ok(a.blk_start, a.blk_len, j, a.M, a.S, a.max_block_len, a.max_query_len);
    malformed = __syncthreads_or(bad);
    if (malformed && tid == 0 && a.status) atomicCAS(a.status, 0, kStatusBadSpans);
    if (tid == 0) a.hdr[1] = malformed;  // for the merge kernel; every CTA writes the same
  } else {
    malformed = a.hdr[1] != 0;
  }
  if (malformed) {  // write nothing
    if (warp == 0) ptx::tmem_dealloc(tmem, kTmemCols);
    return;
  }

  ptx::BoundedWaits waits(kWaitBudget);  // (a wait's mark is its barrier's address: it is in a register there)
  auto wait = [&](int i, uint32_t parity) { waits(bar(i), parity & 1u, (int)bar(i)); };

  int* const job_ring = reinterpret_cast<int*>(smem + kOffJobs);
  const int tok_shift = 7 - a.g_shift, TOK = 1 << tok_shift;  // query tokens of a row tile
  // consumer side of chain x's job ring: copy record number i, release its slot
  auto next_job = [&](int x, uint32_t i) {
    const uint32_t slot = i % kJobRing;
    wait(kJobFull + x * kJobRing + slot, i / kJobRing);
    Job it = read_record(job_ring + (x * kJobRing + slot) * 16);
    if (__any_sync(0xffffffffu, waits.gave_up())) it.flags |= kFStop;  // a wait gave up: the whole warp stops here
    __syncwarp();
    ptx::mbar_arrive_warp(bar(kJobFree + x * kJobRing + slot));
    return it;
  };

  // Registers: 640 x 96 at launch = 256 x 136 (softmax) + 256 x 64 (output) + 128 x 80 (the rest).
  if (warp >= 16) asm volatile("setmaxnreg.dec.sync.aligned.u32 80;");
  if (warp == 19) {
    // ============== padding slots of the output are written as zeros (gaps in front of / behind blocks) ==============
    // (by a warp of its own beside the attention: in front of it, a long ragged grid's 98 MB of zeros were 20 us alone)
    const int per_row = a.N * (HD / 8);
    auto zero_rows = [&](int b, int lo, int hi) {
      __nv_bfloat16* ob = reinterpret_cast<__nv_bfloat16*>(a.o.ptr) + (int64_t)b * a.o.sb;
#pragma unroll 1
      for (int s = lo; s < hi; ++s)
#pragma unroll 4
        for (int i = lane; i < per_row; i += 32)
          *reinterpret_cast<uint4*>(ob + (int64_t)s * a.o.ss + (int64_t)(i / (HD / 8)) * a.o.sh + (i % (HD / 8)) * 8) =
              make_uint4(0, 0, 0, 0);
    };
    // a gap in front of a block: a quarter of it per CTA
    for (int gi = blockIdx.x; gi < a.B * a.M * 4; gi += gridDim.x) {
      const int bm = gi >> 2, part = gi & 3, b = bm / a.M, m = bm % a.M;
      const int32_t* bs = a.blk_start + (size_t)b * a.M;
      const int32_t* bl = a.blk_len + (size_t)b * a.M;
      const int lo = m == 0 ? 0 : bs[m - 1] + bl[m - 1], n = bs[m] - lo;
      zero_rows(b, lo + n * part / 4, lo + n * (part + 1) / 4);
    }
    // The gap behind the last block holds thousands of rows when a batch is padded to its longest prompt: every CTA
    // takes a slice of it.
    for (int b = 0; b < a.B; ++b) {
      const int lo = a.blk_start[(size_t)b * a.M + a.M - 1] + a.blk_len[(size_t)b * a.M + a.M - 1];
      const int rows = a.S - lo;
      if (rows <= 0) continue;
      const int per = (rows + (int)gridDim.x - 1) / (int)gridDim.x;
      const int slot = (int)((blockIdx.x + (unsigned)b) % gridDim.x);
      zero_rows(b, lo + min(rows, slot * per), lo + min(rows, (slot + 1) * per));
    }
  } else if (warp == 16) {
    // =============================== TMA producer ===============================================
    // The whole warp runs the control flow (so addresses and counters stay warp-uniform); one lane
    // issues the copies.
    const bool leader = lane == 0;
    uint32_t n_pub0 = 0, n_pub1 = 0;
    uint32_t out_mask = 0;    // bit s: a load signalled on barrier kKVFull+s has not been handed back yet
    uint32_t free_par = 0;    // bit s: parity of the next kKVFree+s phase
    uint32_t stream_tiles = 0;
    int mode = 0;             // 1 streamed, 2 resident: the two use the slots' barriers differently
    auto publish = [&](int x, const Job& it) {
      const uint32_t np = x ? n_pub1 : n_pub0;
      const uint32_t slot = np % kJobRing;
      if (np >= kJobRing) wait(kJobFree + x * kJobRing + slot, np / kJobRing - 1);
      if (leader && !waits.gave_up()) {  // (behind a wait that gave up the record may still be read)
        if (it.n > 0) {  // its Q tile on its way into L2: the MMA warp requests it when the chain's buffer is free
          ptx::tma_prefetch_4d(&tmQ, 0, it.g * G, it.start + it.t0, it.b);
          if (HD == 128) ptx::tma_prefetch_4d(&tmQ, 64, it.g * G, it.start + it.t0, it.b);
        }
        write_record(job_ring + (x * kJobRing + slot) * 16, it);
        ptx::mbar_arrive(bar(kJobFull + x * kJobRing + slot));  // release: the record is visible to whoever sees the phase flip
      }
      if (x) ++n_pub1; else ++n_pub0;
    };
    // wait until both MMA warps have handed back the load last signalled on barrier s
    auto drain = [&](int s) {
      if ((out_mask >> s) & 1u) {
        wait(kKVFree + s, (free_par >> s) & 1u);
        free_par ^= 1u << s;
        out_mask &= ~(1u << s);
      }
    };
    auto set_mode = [&](int m) {
      if (mode != m) {
#pragma unroll 1
        for (int s = 0; s < kSlots; ++s) drain(s);
        mode = m;
      }
    };
    // K (v = 0) or V (v = 1) of 64 keys starting at token slot `lo` -> pool slot s, completion on barrier `bs`
    auto load_slot = [&](int v, int s, int bs, int g, int b, int lo) {
      const uint32_t dst = sbase + (v ? kOffV : kOffK) + (uint32_t)s * kSlotHalf;
      const CUtensorMap* const tm = v ? &tmV : &tmK;
      ptx::tma_load_4d(dst, tm, bar(kKVFull + bs), 0, g, lo, b);
      if (HD == 128) ptx::tma_load_4d(dst + kPoolHalf, tm, bar(kKVFull + bs), 64, g, lo, b);
    };

    // ---- streamed pair: both chains walk the same 128-key tiles through a two-deep ring (slots 0-1, 2-3) ----
    auto run_pair = [&](int b, int g, int m, int chunk, int p, int start, int len, int s0, int l0, int s2, int l2, int live) {
      Pair pr = decode_pair(a, b, g, m, chunk, p, start, len, s0, l0, s2, l2, live);
      if (!pr.valid) {
        if (a.one_wave && m == a.M - 1 && a.n_split > 1) {
          // a chunk without keys: neutral statistics for its rows (the prologue kernel sets them otherwise)
          const int t1 = min(len, pr.t0_0 + 2 * TOK);
#pragma unroll 1
          for (int i = lane; i < (t1 - pr.t0_0) * G; i += 32)
            a.part_ml[(((int64_t)b * a.N + g * G + (i & (G - 1))) * a.lq_max + pr.t0_0 + (i >> a.g_shift)) * a.n_split + chunk] =
                make_float2(-INFINITY, 0.f);
        }
        return;
      }
      Job& it = pr.job;
      if (a.n_live == nullptr && m == a.M - 1 && m > 0) {  // the query block's context may contain padding slots
        const int32_t* bl = a.blk_len + (size_t)b * a.M;
        int part = 0;
#pragma unroll 1
        for (int i = lane; i < a.M - 1; i += 32) part += bl[i];
        part = __reduce_add_sync(0xffffffffu, part);
        if (part != (it.ctx_hi - it.ctx_lo)) it.flags |= kFCtxCheck;
      }
      set_mode(1);
      const int T = (pr.n_slots + 1) >> 1;
      it.tile0 = (int)(stream_tiles & 1u);
      it.aux = T;
#pragma unroll 1
      for (int x = 0; x < 2; ++x) {
        it.t0 = x ? pr.t0_1 : pr.t0_0;
        it.n = x ? pr.n_1 : pr.n_0;
        publish(x, it);
      }
#pragma unroll 1
      for (int t = 0; t < T; ++t) {
        const int tb = (int)((stream_tiles + (uint32_t)t) & 1u);
        const int nslots = min(2, pr.n_slots - 2 * t);
#pragma unroll 1
        for (int v = 0; v < 2; ++v) {
          drain(2 * tb + v);
          if (leader) {
            ptx::mbar_expect_tx(bar(kKVFull + 2 * tb + v), (uint32_t)nslots * (kSlotBytes / 2));
#pragma unroll 1
            for (int h = 0; h < nslots; ++h) {
              int nk, own_off; bool own;
              int lo = tile_lo(it, 2 * t + h, nk, own, own_off);
              if (!own && (it.flags & kFWindows)) lo = a.win[(size_t)b * a.win_pitch + it.j0 + 2 * t + h].x;
              load_slot(v, 2 * tb + h, 2 * tb + v, g, b, lo);
            }
          }
          out_mask |= 1u << (2 * tb + v);
        }
      }
      stream_tiles += (uint32_t)T;
    };

    // ---- resident block: K/V loaded once, row tiles dealt to the chains largest first ----
    auto run_block = [&](int b, int g, int m, int start, int len, int s0, int l0, bool keep_in, bool keep_out) {
      const int ctx = m > 0 ? l0 : 0;
      const int n_ctx = (ctx + BN - 1) / BN;
      const int ns_blk = n_ctx + (len + BN - 1) / BN;
      const int R = (len + TOK - 1) >> tok_shift;
      const int n_keep = keep_out ? (m > 0 ? n_ctx : (l0 + BN - 1) / BN) : 0;
      set_mode(2);
      int s_next = ns_blk - 1;
      Job it;
      it.b = b; it.g = g; it.m = m; it.chunk = 0;
      it.start = start; it.len = len;
      it.ctx_lo = s0; it.ctx_hi = s0 + ctx; it.n_ctx = n_ctx; it.j0 = 0;
      it.tile0 = 0;
      auto slots_of = [&](int i) { return n_ctx + (min(len, (R - i) * TOK) + BN - 1) / BN; };  // i-th largest tile
      // Deal the row tiles (largest first) to the two chains so that the chains finish together: a tile costs
      // its keys plus a fixed share for writing the output.  Up to 11 tiles every split is tried (the lanes
      // share the 2^(R-1) candidates); beyond that the tiles are dealt 0,1,1,0,0,1,1,0,...
      uint32_t cmask = 0;  // bit i: chain of the i-th largest tile
      if (R <= 11) {
        const int n_cand = 1 << (R - 1);  // tile 0 (the largest) goes to chain 0
        uint32_t best = 0xffffffffu;
#pragma unroll 1
        for (int c = lane; c < n_cand; c += 32) {
          int load0 = 0, load1 = 0;
#pragma unroll 1
          for (int i = 0; i < R; ++i) {
            const int cost = ctx + min(len, (R - i) * TOK) + kTileFixedCost;
            if (((c << 1) >> i) & 1) load1 += cost; else load0 += cost;
          }
          best = min(best, ((uint32_t)max(load0, load1) << 11) | (uint32_t)(c << 1));
        }
        cmask = __reduce_min_sync(0xffffffffu, best) & 0x7ffu;
      } else {
#pragma unroll 1
        for (int i = 0; i < R; ++i) cmask |= (uint32_t)deal_chain(i) << i;
      }
      auto next_same = [&](int i) {  // position of the same chain's next tile, or R
        const uint32_t same = (((cmask >> i) & 1u) ? cmask : ~cmask) & ~((2u << i) - 1u) & ((1u << R) - 1u);
        return same ? __ffs((int)same) - 1 : R;
      };
      const int first1 = (cmask & ((1u << R) - 1u)) ? __ffs((int)cmask) - 1 : R;  // chain 1's first tile (R: none)
      const int s_lo = keep_in ? n_ctx : 0;
#pragma unroll 1
      for (int i = 0; i <= R; ++i) {
        // K/V slots, highest first (the previous block hands them back in that order).  The loop stops at the first slot that is
        // still in use; the block's two largest jobs are published before the producer sleeps on it, so that the chains find
        // their records and request their Q tiles meanwhile (their MMA warps wait for the slots).  (Only those: a ring that
        // filled up with jobs whose K/V cannot be loaded, because the producer sleeps on the ring, would never drain.)
        const bool blocking = i >= 2 || i == R;
#pragma unroll 1
        for (; s_next >= s_lo; --s_next) {
          const int s = s_next;
          if (!blocking && ((out_mask >> s) & 1u) && !__all_sync(0xffffffffu, ptx::mbar_test(bar(kKVFree + s), (free_par >> s) & 1u))) break;
          drain(s);
          const int lo = s < n_ctx ? s0 + s * BN : start + (s - n_ctx) * BN;
          if (leader) {
            ptx::mbar_expect_tx(bar(kKVFull + s), kSlotBytes);
#pragma unroll 1
            for (int v = 0; v < 2; ++v) load_slot(v, s, s, g, b, lo);
          }
          out_mask |= 1u << s;
        }
        const bool tile = i < R;
        if (!tile && first1 < R) break;
        const int x = tile ? (int)((cmask >> i) & 1u) : 1, r = R - 1 - i;  // (no row tile for chain 1: it only hands the slots back)
        it.t0 = tile ? r * TOK : 0;
        it.own_n = tile ? min(len, it.t0 + TOK) : 0;
        it.n = tile ? slots_of(i) : 0;
        const bool first = i == 0 || i == first1;
        const int nx = tile ? next_same(i) : R;
        const int rel_lo = max(n_keep, nx < R ? slots_of(nx) : 0);  // slots kept for the next block are never handed back
        const int rel_hi = first ? ns_blk : it.n;
        it.flags = kFDoc | (first ? kFFirst : 0) | (keep_in ? kFKeep : 0);
        it.aux = rel_lo | (rel_hi << 8);
        publish(x, it);
      }
    };

    // The work list is handed out dynamically: whichever CTA is free claims the next index.  Claims
    // run two items ahead and the block spans of a claimed item one item ahead, so neither the
    // atomic nor the loads are waited for.
    auto claim = [&]() {
      if (a.one_wave) return a.total_items;
      int v = a.total_items;  // (a wait gave up: no more items)
      if (leader && !waits.gave_up()) v = atomicAdd(a.work_counter, 1);
      return (int)gridDim.x + __shfl_sync(0xffffffffu, v, 0);
    };
    int idx = -1, idx_next = blockIdx.x;  // the first item needs no counter: its 0 is item gridDim.x
    ItemRaw raw_next{};
#pragma unroll 1
    while (idx < a.total_items) {
      const int now = idx;
      const ItemRaw raw = raw_next;
      idx = idx_next;
      raw_next = load_item(a, idx, lane);  // in flight while the item before is processed
      idx_next = claim();
      if (now < 0) continue;
      auto fits = [&](int m, int len) {
        const int ctx = m > 0 ? raw.l0 : 0;
        return raw.kind != 0 && (ctx + BN - 1) / BN + (len + BN - 1) / BN <= kSlots;
      };
      bool kept = false;
#pragma unroll 1
      for (int i = 0; i < raw.cnt; ++i) {
        const int m = raw.m + i;
        const int start = __shfl_sync(0xffffffffu, raw.start, i), len = __shfl_sync(0xffffffffu, raw.len, i);
        const int len_nx = __shfl_sync(0xffffffffu, raw.len, (i + 1) & 31);
        if (len <= 0) continue;  // an empty block has no rows
        if (fits(m, len)) {
          const bool keep_out = i + 1 < raw.cnt && len_nx > 0 && fits(m + 1, len_nx) && raw.l0 > 0;
          run_block(raw.b, raw.g, m, start, len, raw.s0, raw.l0, kept, keep_out);
          kept = keep_out;
        } else {
          // the query block's pair and chunk, or a long block's pairs
          const int p1 = raw.kind == 0 ? raw.p + 1 : (len + 2 * TOK - 1) >> (tok_shift + 1);
#pragma unroll 1
          for (int p = raw.kind == 0 ? raw.p : 0; p < p1; ++p)
            run_pair(raw.b, raw.g, m, raw.chunk, p, start, len, raw.s0, raw.l0, raw.s2, raw.l2, raw.live);
        }
      }
    }
    Job stop{};
    stop.flags = kFStop;
#pragma unroll 1
    for (int x = 0; x < 2; ++x) publish(x, stop);
  } else if (warp == 17 || warp == 18) {
    // =============================== MMA issuer of chain x ======================================
    // Whole-warp control flow, one issuing lane (always the same one: tcgen05.commit tracks the
    // MMAs of the thread that executes it).  The two chains' issuers never wait for each other;
    // they only meet in the kKVFree barriers (two arrivals hand a slot back to the TMA warp).
    const int x = warp - 17;
    uint32_t q_uses = 0, p_seen = 0, jobs_done = 0;
    uint32_t full_par = 0;  // bit s: parity of the next kKVFull+s phase this warp has not consumed yet
    int blk_waited = 0;     // resident block: slots [0, blk_waited) have landed
    // Descriptors are built once: every operand buffer has a fixed address, and stepping along K
    // or to another slot only adds a constant to the 16-byte-unit start-address field.
    const uint32_t idesc_pv = ptx::idesc_bf16(BM, HD, 0, 1);
    const uint32_t idesc_qk0 = ptx::idesc_bf16(BM, 0, 0, 0);
    const uint64_t q_desc0 = ptx::smem_desc_sw128(sbase + kOffQ + (uint32_t)x * kQBytes, 16, 1024);
    const uint64_t k_desc0 = ptx::smem_desc_sw128(sbase + kOffK, 16, 1024);
    const uint64_t v_desc0 = ptx::smem_desc_sw128(sbase + kOffV, kPoolHalf, 1024);
    const uint32_t tm_s = tmem + (uint32_t)x * kChainCols, tm_o = tm_s + kColO;
    auto wait_full = [&](int s) {
      wait(kKVFull + s, (full_par >> s) & 1u);
      full_par ^= 1u << s;
    };
    // S = Q K^T against `keys` keys starting at pool slot `slot`
    auto issue_qk = [&](int slot, int keys, bool last) {
      const uint32_t idesc = idesc_qk0 | ((uint32_t)((keys + 15) >> 4) << 18);  // N/8 at bit 17, N a multiple of 16
      const uint32_t a_lo = (uint32_t)q_desc0, a_hi = (uint32_t)(q_desc0 >> 32);
      const uint32_t b_lo = (uint32_t)k_desc0 + (uint32_t)slot * (kSlotHalf >> 4), b_hi = (uint32_t)(k_desc0 >> 32);
      if (ptx::elect_one()) {
#pragma unroll 1
        for (int ks = 0; ks < HD / 16; ++ks) {
          const uint32_t aoff = (uint32_t)(ks >> 2) * ((BM * 128) >> 4) + (uint32_t)(ks & 3) * 2;
          const uint32_t boff = (uint32_t)(ks >> 2) * (kPoolHalf >> 4) + (uint32_t)(ks & 3) * 2;
          ptx::mma_ss_lohi(tm_s, a_lo + aoff, a_hi, b_lo + boff, b_hi, idesc, ks > 0);
        }
        ptx::mma_commit(bar(kSFull + x));
        if (last) ptx::mma_commit(bar(kQFree + x));  // last read of this chain's Q tile
      }
    };
    // O (+)= P V over `keys` keys starting at pool slot `slot`; P sits over the first 64 columns of S (kFine: over all 128)
    auto issue_pv = [&](int slot, int keys, bool first, bool last) {
      const uint32_t b_lo = (uint32_t)v_desc0 + (uint32_t)slot * (kSlotHalf >> 4), b_hi = (uint32_t)(v_desc0 >> 32);
      const int ksteps = (keys + 15) >> 4;
      if (ptx::elect_one()) {
#pragma unroll 1
        for (int ks = 0; ks < BT / 16; ++ks)
          if (ks < ksteps) {
            const uint32_t b_ks = b_lo + (uint32_t)ks * ((16 * 128) >> 4);
            const uint32_t a_ks = tm_s + (kFine ? (uint32_t)(ks >> 2) * 64 + (uint32_t)(ks & 3) * 8 : (uint32_t)ks * 8);
            ptx::mma_ts_lohi(tm_o, a_ks, b_ks, b_hi, idesc_pv, (!first || ks > 0) ? 1u : 0u);
            if (kFine) ptx::mma_ts_lohi(tm_o, a_ks + 32, b_ks, b_hi, idesc_pv, 1u);
          }
        ptx::mma_commit(bar(kPVDone + x));
        if (last) ptx::mma_commit(bar(kOFull + x));
      }
    };
    // keys of a job's last 128-key tile (every earlier tile spans 128 keys: a short context slot inside a
    // tile is masked by the softmax, not trimmed)
    auto last_tile_keys = [&](const Job& jb) {
      const int Tj = (jb.n + 1) >> 1;
      if (Tj == 0) return 0;
      const int cnt = min(2, jb.n - 2 * (Tj - 1));
      int nk, own_off; bool own;
      tile_lo(jb, 2 * (Tj - 1) + cnt - 1, nk, own, own_off);
      return (cnt - 1) * BN + nk;
    };
    // This warp also loads its chain's Q tiles: it is the one that knows when the buffer is free (the job's last
    // Q K^T has completed) and it has nothing else to do at that moment.  q_issued counts the tiles requested;
    // the next job's tile is requested as soon as the current job's last Q K^T is in the pipe and its record
    // has been published, otherwise at the start of that job.
    uint32_t q_issued = 0;
    auto request_q = [&](const Job& jb) {
      if (q_issued > 0) wait(kQFree + x, q_issued - 1);  // every Q K^T of the previous job has read the buffer
      if (ptx::elect_one()) {
        const uint32_t dst = sbase + kOffQ + (uint32_t)x * kQBytes;
        ptx::mbar_expect_tx(bar(kQFull + x), kQBytes);
        ptx::tma_load_4d(dst, &tmQ, bar(kQFull + x), 0, jb.g * G, jb.start + jb.t0, jb.b);
        if (HD == 128) ptx::tma_load_4d(dst + BM * 128, &tmQ, bar(kQFull + x), 64, jb.g * G, jb.start + jb.t0, jb.b);
      }
      ++q_issued;
    };
    // called once the current job's last Q K^T has been issued: request the next job's Q tile if its record is there
    auto request_next_q = [&](uint32_t job_no) {
      if (q_issued != q_uses) return;  // already requested
      const uint32_t nslot = (job_no + 1) % kJobRing;
      if (!__all_sync(0xffffffffu, ptx::mbar_test(bar(kJobFull + x * kJobRing + nslot), ((job_no + 1) / kJobRing) & 1u))) return;
      const Job nxt = read_record(job_ring + (x * kJobRing + nslot) * 16);
      if (!(nxt.flags & kFStop) && nxt.n > 0) request_q(nxt);
    };
    bool pre_qk = false;  // the first Q K^T of the job fetched next is already in the pipe
    for (uint32_t job_no = 0;; ++job_no) {
      const Job it = next_job(x, job_no);
      if (it.flags & kFStop) break;
      const int n = it.n, T = (n + 1) >> 1;
      const int last_keys = last_tile_keys(it);
      auto keys_of = [&](int t) { return t + 1 < T ? BT : last_keys; };
      // (a job whose first Q K^T was issued ahead has had its Q phase consumed there: by now the barrier may be
      // a phase further, and a parity wait must never fall two phases behind)
      if (T > 0 && !pre_qk) {
        if (q_issued == q_uses) request_q(it);  // not requested ahead
        wait(kQFull + x, q_uses);
        ++q_uses;
      }
      if (T == 1 && pre_qk) request_next_q(job_no);  // its only Q K^T went out with the previous job's last P V
      if (it.flags & kFDoc) {
        // ---- resident block: tile t = pool slots 2t, 2t+1; slots land once per block ----
        if (it.flags & kFFirst) blk_waited = (it.flags & kFKeep) ? it.n_ctx : 0;
        auto ensure = [&](int ns) {
#pragma unroll 1
          while (blk_waited < ns) { wait_full(blk_waited); ++blk_waited; }
        };
        if (T > 0) {
          if (!pre_qk) {
            ensure(min(n, 2));
              ptx::tc_fence_after_sync();
            issue_qk(0, keys_of(0), T == 1);
              if (T == 1) request_next_q(job_no);
          }
          pre_qk = false;
          for (int t = 0; t < T; ++t) {
            if (t + 1 < T) ensure(min(n, 2 * t + 4));
            wait(kPFull + x, p_seen);
            ++p_seen;
            if (t == 0 && jobs_done > 0) wait(kOFree + x, jobs_done - 1);
            // After the job's last tile the chain's next row tile of the same block can start at once if its
            // record and its Q tile are already here (its first key tile is resident): its first Q K^T then
            // rides behind this P V, and its S tile is waiting when the softmax warps have drained O.
            Job nxt{};
            bool chain_on = false;
            if (t + 1 == T) {
              const uint32_t nslot = (job_no + 1) % kJobRing;
              if (__all_sync(0xffffffffu, ptx::mbar_test(bar(kJobFull + x * kJobRing + nslot), ((job_no + 1) / kJobRing) & 1u))) {
                nxt = read_record(job_ring + (x * kJobRing + nslot) * 16);
                chain_on = (nxt.flags & kFDoc) && !(nxt.flags & (kFFirst | kFStop)) && nxt.n > 0 &&
                           blk_waited >= min(nxt.n, 2) && q_issued > q_uses &&
                           __all_sync(0xffffffffu, ptx::mbar_test(bar(kQFull + x), q_uses & 1u));
              }
            }
              ptx::tc_fence_after_sync();
            issue_pv(2 * t, keys_of(t), t == 0, t + 1 == T);
            // the chain's next S tile: queued behind the P V that reads P out of the same columns
            if (t + 1 < T) issue_qk(2 * t + 2, keys_of(t + 1), t + 2 == T);
            if (chain_on) {
              const int Tn = (nxt.n + 1) >> 1;
              issue_qk(0, Tn > 1 ? BT : last_tile_keys(nxt), Tn == 1);
              pre_qk = true;
              ++q_uses;  // its Q tile has landed (tested above): that phase is consumed here
            }
              if (t + 2 == T) request_next_q(job_no);  // the job's last Q K^T is in the pipe
          }
          ++jobs_done;
        }
        // hand back the slots no later job of this chain in this block needs
        // (every load of the block is consumed by both issuers, also of slots this chain never reads or
        // that stay resident for the next block: the phase parities must not fall behind)
        const int rel_lo = it.aux & 0xff, rel_hi = (it.aux >> 8) & 0xff;
        ensure(rel_hi);
#pragma unroll 1
        for (int s = rel_lo; s < rel_hi; ++s)
          if (ptx::elect_one()) ptx::mma_commit(bar(kKVFree + s));
      } else {
        // ---- streamed pair: tile t sits in ring position (tile0 + t) & 1 = pool slots 0-1 or 2-3 ----
        const int Ti = it.aux;  // tiles of the item; this chain computes on the first T of them
        auto pos = [&](int t) { return 2 * ((it.tile0 + t) & 1); };
        auto free_kv = [&](int i) {
          if (ptx::elect_one()) ptx::mma_commit(bar(kKVFree + i));
          __syncwarp();
        };
        auto stream_qk = [&](int t) {
          issue_qk(pos(t), keys_of(t), t + 1 == T);
          free_kv(pos(t));
        };
        if (T > 0) {
          wait_full(pos(0));
          ptx::tc_fence_after_sync();
          stream_qk(0);
          if (T == 1) request_next_q(job_no);
        }
        for (int t = 0; t < T; ++t) {
          // (waited for beside the softmax: between P's arrival and the products a wait costs its round trip even when the
          // tile has landed)
          wait_full(pos(t) + 1);
          if (t + 1 < T) wait_full(pos(t + 1));
          wait(kPFull + x, p_seen);
          ++p_seen;
          if (t == 0 && jobs_done > 0) wait(kOFree + x, jobs_done - 1);
          ptx::tc_fence_after_sync();
          issue_pv(pos(t), keys_of(t), t == 0, t + 1 == T);
          free_kv(pos(t) + 1);
          if (t + 1 < T) stream_qk(t + 1);
          if (t + 2 == T) request_next_q(job_no);  // the job's last Q K^T is in the pipe
        }
#pragma unroll 1
        for (int t = T; t < Ti; ++t) {  // not visible to this chain: consume the phases, hand the tile back
          for (int v = 0; v < 2; ++v) {
            wait_full(pos(t) + v);
            free_kv(pos(t) + v);
          }
        }
        if (T > 0) ++jobs_done;
      }
    }
  } else if (warp < 8) {
    // =============================== softmax, chain x ===========================================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 136;");
    const int x = warp >> 2;
    const int r = tid & 127;  // row of the tile = TMEM lane
    const uint32_t tmem_lane = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)x * kChainCols;
    uint32_t s_seen = 0, pv_seen = 0, tiles_done = 0;
    float2* const stat = reinterpret_cast<float2*>(smem + kOffStat) + x * BM;

    for (uint32_t job_no = 0;; ++job_no) {
      const Job it = next_job(x, job_no);
      const int flags = it.flags;
      if (flags & kFStop) break;
      if (it.n == 0) continue;
      const int32_t* bs = a.blk_start + (size_t)it.b * a.M;
      const int32_t* bl = a.blk_len + (size_t)it.b * a.M;
      const int tok = it.t0 + (r >> a.g_shift);
      const bool ctx_check = (flags & kFCtxCheck) != 0;  // the query block's context contains padding slots
      float m_run = -INFINITY, l_run = 0.f;
      const int n_mine = it.n;
      const int t_mine = (n_mine + 1) >> 1;

      for (int t = 0; t < t_mine; ++t) {
        const int cnt = min(2, n_mine - 2 * t);  // slots of this tile the chain sees
        wait(kSFull + x, s_seen);
        ++s_seen;
        if (t > 0) {
          // The previous tile's P V was issued before this tile's Q K^T, so it has completed too: O is stable
          // and the P columns (first half of S) may be overwritten.  Consuming that phase here keeps the pass
          // below free of calls (64 logits are live across its middle).
          wait(kPVDone + x, pv_seen);
          ++pv_seen;
        }
        ptx::tc_fence_after_sync();
        __syncwarp();
        // One pass per 64-key slot: logits -> registers, mask, row maximum, running-max update,
        // p = 2^(s*scale - m) from the same registers, P (bf16) -> columns [32h, 32h+32) of the
        // tile (kFine: [64h, 64h+64)), which only covers logits that have already been consumed.
#pragma unroll 1
        for (int h = 0; h < cnt; ++h) {
          int nk, own_off; bool own;
          const int lo = tile_lo(it, 2 * t + h, nk, own, own_off);
          uint32_t sr[64];
          {
            uint32_t (&lo32)[32] = *reinterpret_cast<uint32_t (*)[32]>(&sr[0]);
            uint32_t (&hi32)[32] = *reinterpret_cast<uint32_t (*)[32]>(&sr[32]);
            ptx::tmem_ld32(tmem_lane + (uint32_t)h * BN, lo32);
            ptx::tmem_ld32(tmem_lane + (uint32_t)h * BN + 32, hi32);
            ptx::tmem_wait_ld(sr);
          }
          // Visibility.  Slots fully inside the visible region need no masking (the common case).
          // Ragged tails and the causal diagonal make columns [0, lim) of a row visible; padded
          // context ranges (reference layout with gaps between blocks) are masked column by column.
          // A masked logit becomes -inf with one select per column, so that its P is exactly 0 and the
          // pass below stays one basic block: skipping the 8-column groups that no row of the warp sees
          // with warp-uniform branches measured 5 % slower over the whole kernel than exponentiating them.
          const bool premasked = !own && ctx_check;  // padded context: columns masked one by one from the slots' validity bits
          if (nk < BN || (own && own_off + BN - 1 > it.t0) || premasked) {  // (warp-uniform)
            const int lim = own ? max(0, min(nk, tok - own_off + 1)) : nk;
            unsigned v0 = lim >= 32 ? ~0u : (1u << lim) - 1u, v1 = lim >= 64 ? ~0u : lim > 32 ? (1u << (lim - 32)) - 1u : 0u;
            if (premasked) {
              // They come with the list of windows; a one-wave call has no list and searches the spans.  (Searching them in
              // every slot, empty ones too, took a grid of 100 documents of 32..256 tokens from 155 to 190 us.)
              if (flags & kFWindows) {
                const int4 w = a.win[(size_t)it.b * a.win_pitch + it.j0 + 2 * t + h];
                v0 &= (unsigned)w.y;
                v1 &= (unsigned)w.z;
              } else {
                v0 &= __ballot_sync(0xffffffffu, slot_valid(bs, bl, a.M, lo + lane));
                v1 &= __ballot_sync(0xffffffffu, slot_valid(bs, bl, a.M, lo + 32 + lane));
              }
            }
#pragma unroll
            for (int c = 0; c < 64; ++c) sr[c] = ((c < 32 ? v0 : v1) & (1u << (c & 31))) ? sr[c] : 0xff800000u;  // -inf: P = 0 exactly
          }
          {
            float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};  // independent chains
#pragma unroll
            for (int c = 0; c < 64; c += 2)
              mx4[(c >> 1) & 3] = ptx::max3(mx4[(c >> 1) & 3], __uint_as_float(sr[c]), __uint_as_float(sr[c + 1]));
            const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * a.scale_log2;  // scale > 0
            float m_new = fmaxf(m_run, mx);
            if (m_run != -INFINITY && m_new - m_run <= kLazy) m_new = m_run;  // keep the old reference: p <= 2^8
            const float m_ref = (m_new == -INFINITY) ? 0.f : m_new;
            const float corr = ptx::ex2(m_run - m_ref);  // 1 when unchanged, 0 on the first visible slot
            const float neg_ref = -m_ref;
            const bool changed = m_new != m_run;
            m_run = m_new;

            // p with packed fp32x2 arithmetic (the warps are bound by instruction issue, not by the special-function unit)
            const ptx::f32x2 sc2 = ptx::pack2(a.scale_log2, a.scale_log2), nr2 = ptx::pack2(neg_ref, neg_ref);
            ptx::f32x2 ps2[2] = {0ull, 0ull};
            uint32_t pk[32], pl[kFine ? 32 : 1];
#pragma unroll
            for (int c = 0; c < 64; c += 4) {
              const ptx::f32x2 t01 = ptx::fma2(ptx::pack2(__uint_as_float(sr[c]), __uint_as_float(sr[c + 1])), sc2, nr2);
              const ptx::f32x2 t23 = ptx::fma2(ptx::pack2(__uint_as_float(sr[c + 2]), __uint_as_float(sr[c + 3])), sc2, nr2);
              float t0, t1, t2, t3;
              ptx::unpack2(t01, t0, t1);
              const float p0 = ptx::ex2(t0), p1 = ptx::ex2(t1);
              ptx::unpack2(t23, t2, t3);
              const float p2 = ptx::ex2(t2), p3 = ptx::ex2(t3);  // (a -inf logit gives exactly 0)
              ps2[1] = ptx::add2(ps2[1], ptx::pack2(p2, p3));
              ps2[0] = ptx::add2(ps2[0], ptx::pack2(p0, p1));
              __nv_bfloat162 h0 = __floats2bfloat162_rn(p0, p1), h1 = __floats2bfloat162_rn(p2, p3);
              pk[c >> 1] = *reinterpret_cast<uint32_t*>(&h0);
              pk[(c >> 1) + 1] = *reinterpret_cast<uint32_t*>(&h1);
              if constexpr (kFine) {
                pl[c >> 1] = low_part(pk[c >> 1], p0, p1);
                pl[(c >> 1) + 1] = low_part(pk[(c >> 1) + 1], p2, p3);
              }
            }
            ptx::tmem_st32(tmem_lane + (uint32_t)h * (kFine ? 64 : 32), pk);
            if constexpr (kFine) ptx::tmem_st32(tmem_lane + (uint32_t)h * 64 + 32, pl);
            if ((t > 0 || h > 0) && __any_sync(0xffffffffu, changed)) {
              // The reference moved by more than the lazy threshold (rare): bring what was accumulated
              // against the old one in line -- O of the earlier tiles, P of this tile's first slot.  (Behind the
              // exponentials, so that the common path from the row maximum to P is one basic block; all of it
              // precedes the arrival that lets the MMA warp read P and add to O.)
              if (t > 0) {
#pragma unroll 1
                for (int ch = 0; ch < HD / 32; ++ch) {
                  uint32_t orow[32];
                  ptx::tmem_ld32(tmem_lane + kColO + (uint32_t)ch * 32, orow);
                  ptx::tmem_wait_ld(orow);
#pragma unroll
                  for (int i = 0; i < 32; ++i) orow[i] = __float_as_uint(__uint_as_float(orow[i]) * corr);
                  ptx::tmem_st32(tmem_lane + kColO + (uint32_t)ch * 32, orow);
                }
              }
              if (h > 0) ptx::tmem_wait_st();  // the first slot's P was stored by this thread: complete before it is read back
              if (kFine && h > 0) {
                uint32_t ph[32], pm[32];
                ptx::tmem_ld32(tmem_lane, ph);
                ptx::tmem_ld32(tmem_lane + 32, pm);
                ptx::tmem_wait_ld(ph);
                ptx::tmem_wait_ld(pm);
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                  const float u = (__uint_as_float(ph[i] << 16) + __uint_as_float(pm[i] << 16)) * corr;
                  const float v = (__uint_as_float(ph[i] & 0xffff0000u) + __uint_as_float(pm[i] & 0xffff0000u)) * corr;
                  const __nv_bfloat162 w = __floats2bfloat162_rn(u, v);
                  ph[i] = *reinterpret_cast<const uint32_t*>(&w);
                  pm[i] = low_part(ph[i], u, v);
                }
                ptx::tmem_st32(tmem_lane, ph);
                ptx::tmem_st32(tmem_lane + 32, pm);
              } else if (h > 0) {
                uint32_t p0[32];
                ptx::tmem_ld32(tmem_lane, p0);
                ptx::tmem_wait_ld(p0);
                const __nv_bfloat162 c2 = __float2bfloat162_rn(corr);  // corr is 1 or at most 2^-8: exact enough in bf16
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                  __nv_bfloat162 v = __hmul2(*reinterpret_cast<__nv_bfloat162*>(&p0[i]), c2);
                  p0[i] = *reinterpret_cast<uint32_t*>(&v);
                }
                ptx::tmem_st32(tmem_lane, p0);
              }
              ptx::tmem_wait_st();
            }
            float s0, s1, s2, s3;
            ptx::unpack2(ps2[0], s0, s1);
            ptx::unpack2(ps2[1], s2, s3);
            l_run = l_run * corr + ((s0 + s1) + (s2 + s3));
          }
        }
        ptx::tmem_wait_st();
        ptx::tc_fence_before_sync();
        __syncwarp();
        ptx::mbar_arrive_warp(bar(kPFull + x));
      }

      ++pv_seen;  // (the output warps wait for the job's last P V)
      if (tiles_done > 0) waits.unless_given_up(bar(kOFree + x), (tiles_done - 1) & 1u, (int)bar(kOFree + x));  // the previous tile's statistics have been read
      ++tiles_done;
      stat[r] = make_float2(m_run, l_run);
      __syncwarp();
      ptx::mbar_arrive_warp(bar(kStat + x));
    }
  } else if (warp < 16) {
    // =============================== output, chain x ============================================
    // O leaves tensor memory and is stored while the chain's softmax warps are at the next row tile already.
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    const int x = (warp >> 2) - 2;
    const int r = tid & 127;  // row of the tile = TMEM lane
    const uint32_t tmem_lane = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)x * kChainCols + kColO;
    const float2* const stat = reinterpret_cast<const float2*>(smem + kOffStat) + x * BM;
    uint32_t done = 0;
    for (uint32_t job_no = 0;; ++job_no) {
      const Job it = next_job(x, job_no);
      if (it.flags & kFStop) break;
      if (it.n == 0) continue;
      const int tok = it.t0 + (r >> a.g_shift);
      const int n = it.g * G + (r & (G - 1));
      const bool active = tok < it.len;
      const bool split = (it.flags & kFSplit) != 0;
      wait(kStat + x, done);
      const float2 ml = stat[r];
      const float m_run = ml.x, l_run = ml.y;
      wait(kOFull + x, done);
      ++done;
      ptx::tc_fence_after_sync();
      auto chunk = [&](int ch, uint32_t (&orow)[32]) {
        __syncwarp();
        ptx::tmem_ld32(tmem_lane + (uint32_t)ch * 32, orow);
        ptx::tmem_wait_ld(orow);
        if (ch + 1 == HD / 32) {  // O is out of TMEM: the next job's first P V may overwrite it
          ptx::tc_fence_before_sync();
          __syncwarp();
          ptx::mbar_arrive_warp(bar(kOFree + x));
        }
      };
      if (split) {
        // un-normalised partial (O, max, sum) of this key chunk; merged by attn_combine_kernel
        const bool wr = active && tok < a.lq_max;
        const int64_t prow = (((int64_t)it.b * a.N + n) * a.lq_max + tok) * a.n_split + it.chunk;
#pragma unroll 1
        for (int ch = 0; ch < HD / 32; ++ch) {
          uint32_t orow[32];
          chunk(ch, orow);
          if (wr) {
            float4* dst = reinterpret_cast<float4*>(a.part_o + prow * HD + ch * 32);
#pragma unroll
            for (int i = 0; i < 8; ++i)
              dst[i] = make_float4(__uint_as_float(orow[4 * i]), __uint_as_float(orow[4 * i + 1]),
                                   __uint_as_float(orow[4 * i + 2]), __uint_as_float(orow[4 * i + 3]));
          }
        }
        if (wr) a.part_ml[prow] = make_float2(m_run, l_run);
      } else {
        // O / l -> bf16, stored straight from registers: each thread owns one 256-byte output row
        // and writes it as 32-byte (full-sector) stores, or 16-byte ones if the output is only 16-byte aligned.
        const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
        __nv_bfloat16* out_row = reinterpret_cast<__nv_bfloat16*>(a.o.ptr) + (int64_t)it.b * a.o.sb +
                                 (int64_t)(it.start + tok) * a.o.ss + (int64_t)n * a.o.sh;
#pragma unroll 1
        for (int ch = 0; ch < HD / 32; ++ch) {
          uint32_t orow[32];
          chunk(ch, orow);
          if (active) {
#pragma unroll
            for (int q8 = 0; q8 < 2; ++q8) {
              uint32_t w[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                __nv_bfloat162 hh = __floats2bfloat162_rn(__uint_as_float(orow[q8 * 16 + 2 * i]) * inv,
                                                          __uint_as_float(orow[q8 * 16 + 2 * i + 1]) * inv);
                w[i] = *reinterpret_cast<uint32_t*>(&hh);
              }
              __nv_bfloat16* dst = out_row + ch * 32 + q8 * 16;
              if (a.o_align32) {
                ptx::st_global_v8(dst, w);
              } else {
                *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
                *reinterpret_cast<uint4*>(dst + 8) = make_uint4(w[4], w[5], w[6], w[7]);
              }
            }
          }
        }
        if (active && a.lse != nullptr)
          a.lse[((int64_t)it.b * a.N + n) * a.S + it.start + tok] = (m_run + log2f(l_run)) * 0.6931471805599453f;
      }
    }
  }

  // ---- teardown ---------------------------------------------------------------------------------
  ptx::tc_fence_before_sync();
  ptx::end_of_waits(waits, [&](int mark) { return wait_code((mark - (int)sBar) >> 3, warp); }, a.status);
  if (warp == 0) ptx::tmem_dealloc(tmem, kTmemCols);
}

}  // namespace

// The kernels' bounded waits (ptx::BoundedWaits) running out, without a fault: one thread waits with a small budget on an
// mbarrier that nothing arrives at, then on another one, which may take one try and must not replace the first one's code,
// then on one whose phase is complete, and leaves as the kernels do.  Anything else than expected is reported as the code
// behind kStatusSelfTest.
__global__ void selftest_wait_kernel(int32_t* status, int budget) {
  __shared__ __align__(8) uint64_t mbar[3];
  uint32_t b[3];
  for (int i = 0; i < 3; ++i) {
    b[i] = ptx::smem_u32(&mbar[i]);
    ptx::mbar_init(b[i], 1);
  }
  ptx::fence_barrier_init();
  ptx::mbar_arrive(b[2]);
  ptx::BoundedWaits waits(budget);
  waits(b[2], 0, kStatusSelfTest + 2);
  bool ok = !waits.gave_up();
  ok &= waits(b[0], 0, kStatusSelfTest) == budget && waits.gave_up();
  ok &= waits(b[1], 0, kStatusSelfTest + 2) == 1;
  ok &= waits(b[2], 0, kStatusSelfTest + 2) == 0 && waits.unless_given_up(b[1], 0, kStatusSelfTest + 2) == 0;
  if (!ok) atomicCAS(status, 0, kStatusSelfTest + 1);
  ptx::end_of_waits(waits, [](int mark) { return mark; }, status);
}

int selftest_wait_launch(int32_t* status, uint32_t budget, cudaStream_t st) {
  selftest_wait_kernel<<<1, 1, 0, st>>>(status, (int)budget);
  BRK_LAUNCHED();
  return BRK_OK;
}

// Launched in front of either attention kernel.  Block 0 checks the block spans (inside [0, S), no longer than
// max_block_len, ordered, not overlapping) and records the verdict in the workspace header -- a non-zero hdr[1]
// makes the attention kernels return without touching memory, and the caller's status word (if any) gets
// kStatusBadSpans.  All blocks reset the work counter and the query block's partial (max, sum) pairs to neutral.  With a
// window list, the last B blocks write it, one prompt each: the 64-slot windows of the query block's context that hold
// any key, {first slot, validity bits}, for prompts with padding between their blocks (a grid of ragged documents: 100
// documents of 32..256 tokens fill 272 of 404 windows).
__device__ void live_windows(const int32_t* bs, const int32_t* bl, int M, int4* win, int* n_live, int pitch) {
  constexpr int kMaxSharedSpans = 2048;
  __shared__ int s_span[2 * kMaxSharedSpans], s_cnt[8], s_sum;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) s_sum = 0;
  __syncthreads();
  int sum = 0;
  for (int i = tid; i < M; i += 256) {
    if (i < M - 1) sum += bl[i];
    if (M <= kMaxSharedSpans) {
      s_span[i] = bs[i];
      s_span[M + i] = bl[i];
    }
  }
  atomicAdd(&s_sum, sum);
  __syncthreads();
  if (M <= kMaxSharedSpans) {
    bs = s_span;
    bl = s_span + M;
  }
  const int lo0 = bs[0], hi = bs[M - 2] + bl[M - 2];
  if (s_sum == hi - lo0) {
    if (tid == 0) *n_live = -1;
    return;
  }
  const int nw = max(0, min(pitch, (hi - lo0 + BN - 1) / BN));
  int base = 0;
  for (int w0 = 0; w0 < nw; w0 += 256) {
    const int lo = lo0 + (w0 + tid) * BN;
    unsigned long long bits = 0;
    if (w0 + tid < nw) {
      int l = 0, h = M;  // first block that starts behind lo
      while (l < h) {
        const int mid = (l + h) >> 1;
        if (bs[mid] <= lo) l = mid + 1; else h = mid;
      }
      for (int m = max(0, l - 1); m < M - 1 && bs[m] < lo + BN; ++m) {
        const int x0 = max(bs[m] - lo, 0), x1 = min(bs[m] + bl[m] - lo, BN);
        if (x1 > x0) bits |= (~0ull >> (BN - (x1 - x0))) << x0;
      }
    }
    const unsigned live = __ballot_sync(0xffffffffu, bits != 0);
    if (lane == 0) s_cnt[warp] = __popc(live);
    __syncthreads();
    int at = base + __popc(live & ((1u << lane) - 1u));
    for (int i = 0; i < 8; ++i) {
      if (i < warp) at += s_cnt[i];
      base += s_cnt[i];
    }
    if (bits != 0) win[at] = make_int4(lo, (int)(unsigned)bits, (int)(unsigned)(bits >> 32), 0);
    __syncthreads();
  }
  if (tid == 0) *n_live = base;
}

__global__ void __launch_bounds__(256) attn_prologue_kernel(const int32_t* __restrict__ blk_start, const int32_t* __restrict__ blk_len, int B,
                                     int M, int S, int max_block_len, int max_query_len, int* hdr, int32_t* status,
                                     float2* ml, int64_t n_ml, int4* win, int* n_live, int win_pitch) {
  if (win != nullptr && blockIdx.x >= gridDim.x - B) {
    const int b = blockIdx.x - (gridDim.x - B);
    live_windows(blk_start + (size_t)b * M, blk_len + (size_t)b * M, M, win + (size_t)b * win_pitch, n_live + b, win_pitch);
    return;
  }
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n_ml) ml[i] = make_float2(-INFINITY, 0.f);
  if (blockIdx.x != 0) return;
  __shared__ int bad;
  if (threadIdx.x == 0) {
    bad = 0;
    hdr[0] = 0;
  }
  __syncthreads();
  for (int j = threadIdx.x; j < B * M; j += blockDim.x) {
    const bool ok = span_ok(blk_start, blk_len, j, M, S, max_block_len, max_query_len);
    if (!ok) bad = 1;  // benign race: every writer stores the same value
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    hdr[1] = bad;
    if (bad && status) atomicCAS(status, 0, kStatusBadSpans);
  }
}

int attn_prologue_launch(const brk_attn_params& p, int* hdr, float2* ml, int64_t n_ml, int4* win, int* n_live, int win_pitch,
                         cudaStream_t st) {
  const unsigned blocks = (unsigned)(n_ml > 0 ? (n_ml + 255) / 256 : 1) + (win ? p.B : 0);
  attn_prologue_kernel<<<blocks, 256, 0, st>>>(p.blk_start, p.blk_len, p.B, p.M, p.S, p.max_block_len, p.max_query_len,
                                               hdr, p.status, ml, n_ml, win, n_live, win_pitch);
  BRK_LAUNCHED();
  return BRK_OK;
}

// Key chunks for the query block.  Its context is every earlier token of the prompt (S is the only
// bound known on the host), walked 128 keys per step per row tile, 2.3 us each; cutting it into chunks of about
// 1024 keys keeps that serial chain short and spreads it over the SMs.  A call whose chunks of 1024 keys leave more than a
// third of the SMs idle, with other blocks for no more than one and a half rounds of them, is cut further, down to 256 keys,
// while the chunks find idle SMs (one prompt of 8 documents of 100 tokens 31.1 -> 20.6 us, of 20 documents of 160 tokens 51.7 ->
// 41.3, 2 prompts of 8 documents of 500 tokens 182 -> 119; with more blocks the finer chunks cost: 2 prompts of 20 documents
// 68.8 -> 75.8, one of 50 74.1 -> 78.7); below 640 slots the chain is shorter than the merge.
// The rule decides the order in which a row's keys are summed, so it does not chase the last chunk: batches cut into one chunk
// per SM instead (4 prompts of 100 documents: 5 of each, not 16) differ in the last bit of a few outputs, which 20 layers of
// the 7B ranker turn into 2.4e-3 of its logits, for 451 us where this takes 459.
static int tc_splits(const brk_attn_params& p) {
  if (p.M < 2) return 1;
  const int G = std::max(1, p.N / std::max(1, p.Nk));
  int n = std::max(1, std::min(32, (p.S + 1023) / 1024));
  if (p.S > 640) {
    const int tok2 = std::max(1, 2 * BM / G);
    const int64_t pairs = (int64_t)p.B * p.Nk * ((query_rows(p) + tok2 - 1) / tok2);
    const int64_t blocks = (int64_t)p.B * p.Nk * (p.M - 1);
    if (3 * pairs * n <= 2 * sm_count() && 2 * blocks <= 3 * sm_count())
      n = std::max(n, (int)std::min<int64_t>(std::min(32, (p.S + 255) / 256), sm_count() / std::max<int64_t>(1, pairs)));
  }
  return p.D == 128 && G == 4 ? n : capped_chunks(p, n);  // (there the chunks are never fewer: see above)
}

// Header (work counter, span verdict), live windows of the query block's context, partials of its key chunks.
static int win_pitch(const brk_attn_params& p) { return p.S / BN + 1; }
static size_t window_bytes(const brk_attn_params& p) {
  return ((size_t)p.B * (win_pitch(p) * sizeof(int4) + sizeof(int)) + 255) & ~(size_t)255;
}
size_t attn_tc_workspace(const brk_attn_params& p) {
  const int ns = tc_splits(p);
  const size_t rows = ns > 1 ? (size_t)p.B * p.N * query_rows(p) * ns : 0;
  return kWsHeader + window_bytes(p) + rows * (p.D * sizeof(float) + sizeof(float2));
}

template <int HD, bool kFine>
static int attn_tc_run(const brk_attn_params& p, void* ws, size_t ws_bytes, cudaStream_t st) {
  const int G = p.N / p.Nk;
  BRK_REQUIRE(G == 1 || G == 2 || G == 4 || G == 8, BRK_E_UNSUPPORTED, "tcgen05 attention needs N/Nk in {1,2,4,8}, got %d", G);
  BRK_REQUIRE(p.scale > 0.f, BRK_E_ARG, "softmax scale must be positive");
  const int ns = tc_splits(p);
  const size_t need = attn_tc_workspace(p);
  BRK_REQUIRE(ws != nullptr && ws_bytes >= need && ((uintptr_t)ws & 15) == 0, BRK_E_WORKSPACE,
              "attention workspace: %zu bytes (16-byte aligned) needed, %zu given", need, ws_bytes);
  int gs = 0;
  while ((1 << gs) < G) ++gs;
  const int TOK = BM / G;
  const int lq = query_rows(p);
  const int pairs_q = (lq + 2 * TOK - 1) / (2 * TOK);
  const int64_t nbg = (int64_t)p.B * p.Nk;
  CUtensorMap tq, tk, tv;
  int rc;
  if ((rc = make_tmap_bf16(&tq, p.q.ptr, HD, p.N, p.S, p.B, p.q.stride_h, p.q.stride_s, p.q.stride_b, G, TOK))) return rc;
  if ((rc = make_tmap_bf16(&tk, p.k.ptr, HD, p.Nk, p.S, p.B, p.k.stride_h, p.k.stride_s, p.k.stride_b, 1, BN))) return rc;
  if ((rc = make_tmap_bf16(&tv, p.v.ptr, HD, p.Nk, p.S, p.B, p.v.stride_h, p.v.stride_s, p.v.stride_b, 1, BN))) return rc;
  static std::atomic<int> sms[64] = {};  // SMs of a device whose kernel is configured (by any thread: the steps can be repeated)
  int dev = 0;
  BRK_CUDA(cudaGetDevice(&dev));
  BRK_REQUIRE(dev >= 0 && dev < 64, BRK_E_UNSUPPORTED, "device ordinal %d out of range", dev);
  int n_sm = sms[dev].load(std::memory_order_acquire);
  if (n_sm == 0) {
    BRK_CUDA(cudaFuncSetAttribute(attn_tc_kernel<HD, kFine>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)Geo<HD>::kSmemBytes));
    n_sm = sm_count();
    BRK_REQUIRE(n_sm > 0, BRK_E_CUDA, "could not read the SM count");
    sms[dev].store(n_sm, std::memory_order_release);
  }
  // Blocks are handed out in groups of consecutive blocks of one (prompt, KV head), so that the prefix's K/V
  // stays in shared memory from one block to the next.  Balance matters more than that reuse (measured: single
  // blocks 0.560 ms, groups of three 0.572 ms on 4 prompts of 100 documents), so groups only form when every SM
  // still gets two dozen of them.
  int group = (int)((nbg * (p.M > 1 ? p.M - 1 : 0)) / (24 * (int64_t)n_sm));
  group = group < 1 ? 1 : (group > kMaxGroup ? kMaxGroup : group);
  const int n_groups = p.M > 1 ? (p.M - 1 + group - 1) / group : 0;
  const int64_t sec1 = nbg * ns * pairs_q;
  const int64_t total_items = sec1 + nbg * n_groups;
  BRK_REQUIRE(total_items < (1ll << 30), BRK_E_UNSUPPORTED, "too many work items (%lld)", (long long)total_items);
  TcArgs a;
  a.o = make_view(p.o);
  a.lse = p.lse;
  a.blk_start = p.blk_start;
  a.blk_len = p.blk_len;
  a.status = p.status;
  a.hdr = reinterpret_cast<int*>(ws);
  a.B = p.B; a.N = p.N; a.Nk = p.Nk; a.S = p.S; a.M = p.M;
  a.G = G; a.g_shift = gs;
  a.scale_log2 = p.scale * 1.4426950408889634f;
  a.n_split = ns;
  a.lq_max = lq;
  a.pairs_q = pairs_q;
  a.group = group;
  a.n_groups = n_groups;
  a.o_align32 = (((uintptr_t)p.o.ptr & 31) == 0 && p.o.stride_b % 16 == 0 && p.o.stride_h % 16 == 0 && p.o.stride_s % 16 == 0) ? 1 : 0;
  a.sec1 = (int)sec1;
  a.total_items = (int)total_items;
  a.div_sec1 = make_fastdiv((uint32_t)(nbg * ns));
  a.div_nbg = make_fastdiv((uint32_t)nbg);
  a.div_nk = make_fastdiv((uint32_t)p.Nk);
  const size_t rows = (size_t)p.B * p.N * lq * ns;
  int4* const win = reinterpret_cast<int4*>(static_cast<uint8_t*>(ws) + kWsHeader);
  float* const part = reinterpret_cast<float*>(static_cast<uint8_t*>(ws) + kWsHeader + window_bytes(p));
  a.work_counter = reinterpret_cast<int*>(ws);
  a.part_o = ns > 1 ? part : nullptr;
  a.part_ml = ns > 1 ? reinterpret_cast<float2*>(part + rows * HD) : nullptr;
  // A call whose items all start at once needs neither the counter nor the partials' reset: its CTAs check the spans
  // themselves.  (One prompt of 5 documents: the prologue kernel and the gap behind it were 4 of 20 us.)
  a.max_block_len = p.max_block_len;
  a.max_query_len = p.max_query_len;
  a.one_wave = total_items <= n_sm;
  a.win = nullptr;
  a.n_live = nullptr;
  a.win_pitch = win_pitch(p);
  if (!a.one_wave) {
    int* const n_live = reinterpret_cast<int*>(win + (size_t)p.B * a.win_pitch);
    const bool list = p.M > 2;  // (a single block has no gaps)
    if (list) {
      a.win = win;
      a.n_live = n_live;
    }
    if ((rc = attn_prologue_launch(p, reinterpret_cast<int*>(ws), a.part_ml, ns > 1 ? (int64_t)rows : 0, list ? win : nullptr, n_live,
                                   a.win_pitch, st)))
      return rc;
  }
  const int grid = (int)(total_items < n_sm ? total_items : n_sm);
  if ((rc = launch_dependent(attn_tc_kernel<HD, kFine>, dim3(grid), dim3(kThreads), Geo<HD>::kSmemBytes, st, tq, tk, tv, a))) return rc;
  if (ns > 1) {
    const CombineArgs c{a.o, a.lse, a.blk_start, a.blk_len, a.hdr, p.B, p.N, p.S, p.M, lq, ns, a.part_o, a.part_ml};
    return attn_combine_launch<__nv_bfloat16, HD>(c, st);
  }
  return BRK_OK;
}

int attn_tc_launch(const brk_attn_params& p, void* ws, size_t ws_bytes, cudaStream_t st) {
  BRK_REQUIRE(p.dtype == BRK_BF16 && (p.D == 64 || p.D == 128), BRK_E_UNSUPPORTED,
              "tcgen05 attention needs bf16 and head_dim 64 or 128 (dtype %d, head_dim %d)", p.dtype, p.D);
  // AUTO keeps the precision of the kernel it would choose otherwise; asked for by name, this kernel rounds P to bf16.
  const bool fine = p.algo == BRK_ALGO_AUTO && !(p.D == 128 && p.Nk > 0 && p.N / p.Nk == 4);
  if (p.D == 128) return fine ? attn_tc_run<128, true>(p, ws, ws_bytes, st) : attn_tc_run<128, false>(p, ws, ws_bytes, st);
  return fine ? attn_tc_run<64, true>(p, ws, ws_bytes, st) : attn_tc_run<64, false>(p, ws, ws_bytes, st);
}

}  // namespace brk
