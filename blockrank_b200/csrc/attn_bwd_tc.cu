// BlockRank attention backward on the sm_100a tensor cores (tcgen05 + TMEM), bf16, head_dim 64 or 128.
//
// A work item is one block of one (prompt, KV head): the keys are the block's own ones, for a document with the prefix
// block's in front, in tiles of 128; the rows are the block's own query tokens (all G heads of the group, 128 / G tokens
// x G heads per row tile) and then the query block's rows, which see the block's own keys.  So every key of a document
// and every row of a document meets all its partners inside one item:
//
//   dV, dK of own keys     accumulate in tensor memory over the key tile's row tiles and are stored once, in bf16
//   dK, dV of the prefix   get one fp32 reduction per document item
//   dQ of own rows         is the sum over the item's key tiles: two at most for documents up to 128 tokens plus prefix;
//                          a partial sum waits in fp32 in a scratch of the CTA, laid out for coalesced access by the
//                          thread that wrote it
//   dQ of the query block  fp32 reductions (every item contributes)
//
// Outputs leave through shared memory by TMA (store or fp32 add), 32 rows per warp.
//
// Per (key tile, row tile) pair, all five products on tcgen05, keys down the 128 TMEM lanes:
//   S^T = K Q^T      dP^T = V dO^T      P^T = 2^(S^T scale - lse)     dS^T = P^T (dP^T - delta)
//   dV += P^T dO (P^T read from tensor memory)    dK += dS^T Q    dQ = dS K   (dS^T in shared memory serves both: K-major
//                                                 for dK, MN-major for dQ)
//
// Roles (512 threads, one CTA per SM, items claimed from a global counter, longest blocks first):
//   warps 0-7   element-wise part: warp w owns lanes 32 (w % 4) and the row-tile columns 64 (w / 4) + {0..63}; between key
//               tiles they load K / V (cp.async, zero beyond the list, so any prefix length packs against any document)
//   warps 8-11  outputs: dQ after every pair, dV and dK after every key tile, from tensor memory through shared memory to
//               TMA, beside the element-wise part of the next pair
//   warp 12     MMA issue
//   warp 13     claims items, loads Q (two stages) and dO (one) by TMA and the columns' lse and delta
//   warps 14-15 zero the rows of a partial row tile that lie beyond its block
//
// Order of the tensor pipe: dP(i) | dV(i) S(i+1) | dQ(i) dK(i): the exponentials of tile i + 1 run beside dQ(i) / dK(i) and
// the dS of tile i beside dV(i) / S(i+1).  Tensor memory (head_dim 128, all 512 columns): S / P 128, dP / dQ 128, dV 128,
// dK 128; dQ shares dP's columns, so the way dQ(i) -> read out -> dP(i+1) -> dS(i+1) is the kernel's cycle, and that is
// why the reading has warps of its own.
#include <cuda.h>

#include <algorithm>

#include "brk_common.cuh"
#include "mma_bf16.cuh"
#include "tc_ptx.cuh"

namespace brk {

namespace {

constexpr int kTile = 128;  // keys per key tile, rows per row tile
constexpr int kThreads = 512;
constexpr uint32_t kChunk = kTile * 128;  // 128 rows of 64 bf16: one 64-wide chunk of a tile
constexpr int kWaitBudget = 1 << 18;
constexpr int kMaxRowTiles = 16;  // per block: bounds the dQ scratch of a CTA (64 KB per tile at head_dim 128)

template <int HD>
struct Geo {
  static constexpr uint32_t kTileBytes = (HD / 64) * kChunk;
  static constexpr uint32_t kOffK = 0;
  static constexpr uint32_t kOffV = kOffK + kTileBytes;
  static constexpr uint32_t kOffQ = kOffV + kTileBytes;  // two stages
  static constexpr uint32_t kOffG = kOffQ + 2 * kTileBytes;
  static constexpr uint32_t kOffDs = kOffG + kTileBytes;
  static constexpr uint32_t kOffOut = kOffDs + 2 * kChunk;   // output staging: two slabs of 4 KB for each of warps 8-11
  static constexpr uint32_t kOffCol = kOffOut + 8 * 4096;    // two stages of [-lse log2 e | delta], 128 floats each
  static constexpr uint32_t kOffBar = kOffCol + 2 * 2 * kTile * 4;
  static constexpr uint32_t kSmem = kOffBar + 256;
  static_assert(kSmem <= 232448, "shared memory per CTA");
};
constexpr uint32_t kColS = 0, kColDp = 128, kColDv = 256, kColDk = 384;

enum {
  kQFull = 0,    // +stage  Q landed and the columns' lse / delta written (expect_tx arrival + 1)
  kQFree = 2,    // +stage  dK has read the stage (commit + 2 warps)
  kQTail = 4,    // +stage  the rows beyond the block zeroed in a partial Q tile (2 warps).  Per stage: with one barrier the
                 //         two tiles behind a key tile's end could both arrive before the first was waited for
  kGFull = 6,    // dO landed
  kGFree = 7,    // dV has read it (commit + 2 warps)
  kGTail = 8,    // as kQTail
  kSFull = 9,
  kDpFull = 10,
  kPFull = 11,   // P^T in tensor memory (8 warps)
  kDsFull = 12,  // dS^T in shared memory, dP consumed (8 warps)
  kDqFull = 13,
  kDqFree = 14,  // dQ read out (4 warps)
  kAccFull = 15, // every product of the key tile complete
  kAccFree = 16, // dV, dK read out (4 warps)
  kKvFull = 17,  // K, V of the key tile in shared memory (8 warps)
  kItemFull = 18,  // +slot
  kItemFree = 20,  // +slot (15 consuming warps)
  kNumBars = 22
};
static_assert(kNumBars * 8 + 16 <= 256, "barrier area");  // + TMEM base, two item slots

struct BwdTcArgs {
  View q, k, v, o, d_o, dq, dk, dv;
  const float* lse;
  float* delta;     // [B, N, S]
  float* pre;       // prefix accumulators: dK then dV, [B, Nk, max_block_len, D] each; nullptr: block 0 stored directly
  float* dq32;      // [B, N, max_block_len, D]: dQ of the last block's rows
  float* part;      // [CTA][row tile][HD / 4][128 threads] float4: dQ of rows whose keys span several tiles
  int* counter;
  int* order;       // (prompt, block) pairs, longest block first; nullptr: as they come
  int32_t* status;
  const int32_t* blk_start;
  const int32_t* blk_len;
  int B, N, Nk, S, M, G, g_shift, max_block_len, row_tiles, total_items;
  float scale, scale_log2;
};

__device__ __forceinline__ void span_of(const BwdTcArgs& a, int b, int m, int& start, int& len) {
  start = a.blk_start[(size_t)b * a.M + m];
  len = a.blk_len[(size_t)b * a.M + m];
  if (start < 0 || len < 0 || len > a.max_block_len || start > a.S - len) len = 0;  // skipped: nothing out of bounds
}

struct Item {
  int b, g, m;
  int start, len;    // the block
  int s0, l0;        // prefix keys in front of the own ones (l0 = 0: none)
  int qs, ql;        // query-block rows that see the own keys (ql = 0: none)
  int n_kt, R, RQ;   // key tiles, own row tiles, query row tiles
};

__device__ __forceinline__ Item decode(const BwdTcArgs& a, int idx) {
  Item it;
  const int bm = a.order ? a.order[idx / a.Nk] : idx / a.Nk;
  it.b = bm / a.M;
  it.m = bm % a.M;
  it.g = idx % a.Nk;
  span_of(a, it.b, it.m, it.start, it.len);
  it.s0 = it.l0 = it.qs = it.ql = 0;
  if (it.m > 0 && it.m < a.M - 1) span_of(a, it.b, 0, it.s0, it.l0);
  if (it.m < a.M - 1) span_of(a, it.b, a.M - 1, it.qs, it.ql);
  const int tok = kTile >> a.g_shift;
  it.n_kt = it.len > 0 ? (it.l0 + it.len + kTile - 1) / kTile : 0;
  it.R = (it.len + tok - 1) / tok;
  it.RQ = (it.ql + tok - 1) / tok;
  return it;
}

// Row tiles of key tile kt: own tiles r0 .. R-1, then query tiles 0 .. nq-1.
struct RowList {
  int r0, n_own, n;
};
__device__ __forceinline__ RowList rows_of(const BwdTcArgs& a, const Item& it, int kt) {
  RowList l;
  l.r0 = max(0, kt * kTile - it.l0) >> (7 - a.g_shift);  // first tile with a token at or behind the key tile's first own key
  l.n_own = it.R - l.r0;
  l.n = l.n_own + ((kt + 1) * kTile > it.l0 ? it.RQ : 0);
  return l;
}
struct RowTile {
  bool own;
  int t0, nrow, slot;  // first token inside the block, valid rows, first token slot
  int r;               // own: row tile number
};
__device__ __forceinline__ RowTile row_tile(const BwdTcArgs& a, const Item& it, const RowList& l, int i) {
  RowTile t;
  t.own = i < l.n_own;
  t.r = t.own ? l.r0 + i : i - l.n_own;
  t.t0 = t.r * (kTile >> a.g_shift);
  t.slot = (t.own ? it.start : it.qs) + t.t0;
  t.nrow = min(kTile, ((t.own ? it.len : it.ql) - t.t0) << a.g_shift);
  return t;
}

// Inputs by row tile; outputs by warp (32 rows or keys).
struct Maps {
  CUtensorMap q, g;        // Q, dO: box {64, G, 128 / G}
  CUtensorMap dq, dk, dv;  // boxes {64, G, 32 / G}, {64, 1, 32}
  CUtensorMap dq32, pre;   // fp32 sums: boxes {32, G, 32 / G}, {32, 1, 32}
};

template <int HD>
__global__ void __launch_bounds__(kThreads, 1) attn_bwd_tc_kernel(const __grid_constant__ Maps maps, const BwdTcArgs a) {
  using L = Geo<HD>;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sbase = ptx::smem_u32(smem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  auto bar = [&](int i) { return sbase + L::kOffBar + (uint32_t)i * 8u; };
  uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(smem + L::kOffBar + kNumBars * 8);
  int* const item_slot = reinterpret_cast<int*>(smem + L::kOffBar + kNumBars * 8 + 4);
  if (tid == 0) {
    for (int i = 0; i < kNumBars; ++i) {
      uint32_t cnt = 1u;
      if (i == kPFull || i == kDsFull || i == kKvFull) cnt = 8u;
      if (i == kDqFree || i == kAccFree) cnt = 4u;
      if (i == kQFull || i == kQFull + 1 || i == kQTail || i == kQTail + 1 || i == kGTail) cnt = 2u;
      if (i == kQFree || i == kQFree + 1 || i == kGFree) cnt = 3u;
      if (i >= kItemFree) cnt = 15u;
      ptx::mbar_init(bar(i), cnt);
    }
    ptx::fence_barrier_init();
    ptx::prefetch_tmap(&maps.q);
    ptx::prefetch_tmap(&maps.g);
  }
  __syncwarp();
  if (warp == 0) {
    ptx::tmem_alloc(ptx::smem_u32(tmem_slot), 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  ptx::BoundedWaits waits(kWaitBudget);
  auto wait = [&](int i, uint32_t parity, int code) { waits(bar(i), parity & 1u, code); };
  auto arrive = [&](int i) {
    __syncwarp();
    ptx::mbar_arrive_warp(bar(i));
  };
  uint32_t n_items = 0;
  // next item of this CTA, or -1 (every warp but the loader)
  auto next_item = [&]() {
    const uint32_t slot = n_items & 1u;
    wait(kItemFull + slot, n_items >> 1, 60);
    int idx = item_slot[slot];
    if (__any_sync(0xffffffffu, waits.gave_up())) idx = -1;
    arrive(kItemFree + slot);
    ++n_items;
    return idx;
  };

  // Registers: 512 x 128 at launch = 256 x 136 + 128 x 176 + 128 x 64.
  if (warp >= 12) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    if (warp == 13) {
      // =============================== loader ====================================================
      uint32_t tile = 0, pub = 0;
      const bool leader = lane == 0;
      for (;;) {
        int idx = 0;
        if (leader) idx = atomicAdd(a.counter, 1);
        idx = __shfl_sync(0xffffffffu, idx, 0);
        if (idx >= a.total_items) idx = -1;
        if (pub >= 2) wait(kItemFree + (pub & 1u), (pub >> 1) - 1, 61);
        if (leader) {
          item_slot[pub & 1u] = idx;
          ptx::mbar_arrive(bar(kItemFull + (pub & 1u)));
        }
        ++pub;
        if (idx < 0 || __any_sync(0xffffffffu, waits.gave_up())) break;
        const Item it = decode(a, idx);
        for (int kt = 0; kt < it.n_kt; ++kt) {
          const RowList rows = rows_of(a, it, kt);
          for (int i = 0; i < rows.n; ++i, ++tile) {
            const RowTile t = row_tile(a, it, rows, i);
            const uint32_t st = tile & 1u;
            if (tile >= 2) wait(kQFree + st, (tile >> 1) - 1, 62);
            if (leader) {
              const uint32_t q = sbase + L::kOffQ + st * L::kTileBytes;
              ptx::mbar_expect_tx(bar(kQFull + st), L::kTileBytes);
#pragma unroll
              for (int c = 0; c < HD / 64; ++c)
                ptx::tma_load_4d(q + c * kChunk, &maps.q, bar(kQFull + st), 64 * c, it.g * a.G, t.slot, it.b);
            }
            float* const col = reinterpret_cast<float*>(smem + L::kOffCol) + st * 2 * kTile;
#pragma unroll
            for (int j = 0; j < kTile / 32; ++j) {
              const int c = lane + 32 * j;
              float nl = -INFINITY, dl = 0.f;  // beyond the block: P = 0
              if (c < t.nrow) {
                const size_t id = ((size_t)it.b * a.N + it.g * a.G + (c & (a.G - 1))) * a.S + t.slot + (c >> a.g_shift);
                nl = a.lse[id] * -1.4426950408889634f;
                dl = a.delta[id];
              }
              col[c] = nl;
              col[kTile + c] = dl;
            }
            arrive(kQFull + st);
            if (tile >= 1) wait(kGFree, tile - 1, 63);
            if (leader) {
              ptx::mbar_expect_tx(bar(kGFull), L::kTileBytes);
#pragma unroll
              for (int c = 0; c < HD / 64; ++c)
                ptx::tma_load_4d(sbase + L::kOffG + c * kChunk, &maps.g, bar(kGFull), 64 * c, it.g * a.G, t.slot, it.b);
            }
          }
        }
      }
    } else if (warp == 12) {
      // =============================== MMA issue =================================================
      uint32_t tile = 0, kts = 0, q_tails0 = 0, q_tails1 = 0, g_tails = 0;
      const uint32_t id_dkv = ptx::idesc_bf16(kTile, HD, 0, 1);  // dV, dK: A K-major, B (dO / Q) MN-major
      const uint32_t id_dq = ptx::idesc_bf16(kTile, HD, 1, 1);   // dQ: A (dS) and B (K) MN-major
      const uint64_t k_k = ptx::smem_desc_sw128(sbase + L::kOffK, 16, 1024), v_k = ptx::smem_desc_sw128(sbase + L::kOffV, 16, 1024);
      const uint64_t k_mn = ptx::smem_desc_sw128(sbase + L::kOffK, kChunk, 1024);
      const uint64_t ds_k = ptx::smem_desc_sw128(sbase + L::kOffDs, 16, 1024), ds_mn = ptx::smem_desc_sw128(sbase + L::kOffDs, kChunk, 1024);
      const uint64_t q_k = ptx::smem_desc_sw128(sbase + L::kOffQ, 16, 1024), q_mn = ptx::smem_desc_sw128(sbase + L::kOffQ, kChunk, 1024);
      const uint64_t g_k = ptx::smem_desc_sw128(sbase + L::kOffG, 16, 1024), g_mn = ptx::smem_desc_sw128(sbase + L::kOffG, kChunk, 1024);
      constexpr uint32_t kStage = L::kTileBytes >> 4;
      // contraction over head_dim: both operands K-major, [128 rows][64] chunks
      auto nt = [&](uint32_t d, uint64_t da, uint64_t db, uint32_t boff, int n16) {
        const uint32_t idesc = ptx::idesc_bf16(kTile, 0, 0, 0) | ((uint32_t)n16 << 18);
#pragma unroll
        for (int ks = 0; ks < HD / 16; ++ks) {
          const uint32_t off = (uint32_t)(ks >> 2) * (kChunk >> 4) + (uint32_t)(ks & 3) * 2;
          ptx::mma_ss_lohi(d, (uint32_t)da + off, (uint32_t)(da >> 32), (uint32_t)db + boff + off, (uint32_t)(db >> 32), idesc, ks > 0);
        }
      };
      for (;;) {
        const int idx = next_item();
        if (idx < 0) break;
        const Item it = decode(a, idx);
        for (int kt = 0; kt < it.n_kt; ++kt, ++kts) {
          const RowList rows = rows_of(a, it, kt);
          const int keys16 = (min(kTile, it.l0 + it.len - kt * kTile) + 15) >> 4;
          wait(kKvFull, kts, 64);
          auto issue_s = [&](uint32_t no, int i) {  // S^T of row tile i (tile number no)
            const RowTile t = row_tile(a, it, rows, i);
            wait(kQFull + (no & 1u), no >> 1, 65);
            if (t.nrow < kTile) wait(kQTail + (no & 1u), (no & 1u) ? q_tails1++ : q_tails0++, 66);
            ptx::tc_fence_after_sync();
            if (ptx::elect_one()) {
              nt(tmem + kColS, k_k, q_k, (no & 1u) * kStage, (t.nrow + 15) >> 4);
              ptx::mma_commit(bar(kSFull));
            }
          };
          for (int i = 0; i < rows.n; ++i, ++tile) {
            const RowTile t = row_tile(a, it, rows, i);
            const uint32_t so = (tile & 1u) * kStage;
            const int r16 = (t.nrow + 15) >> 4;
            if (i == 0) issue_s(tile, 0);
            wait(kGFull, tile, 67);
            if (t.nrow < kTile) wait(kGTail, g_tails++, 68);
            if (tile > 0) wait(kDqFree, tile - 1, 69);  // dQ of the previous tile has left these columns
            ptx::tc_fence_after_sync();
            if (ptx::elect_one()) {
              nt(tmem + kColDp, v_k, g_k, 0, r16);
              ptx::mma_commit(bar(kDpFull));
            }
            wait(kPFull, tile, 70);
            if (i == 0 && kts > 0) wait(kAccFree, kts - 1, 71);  // dV and dK of the previous key tile have been read out
            ptx::tc_fence_after_sync();
            if (ptx::elect_one()) {  // dV += P^T dO: each warp group wrote its 64 columns of P over the first half of its columns of S
              for (int ks = 0; ks < r16; ++ks)
                ptx::mma_ts_lohi(tmem + kColDv, tmem + kColS + (uint32_t)(ks >> 2) * 64 + (uint32_t)(ks & 3) * 8,
                                 (uint32_t)g_mn + (uint32_t)ks * 128, (uint32_t)(g_mn >> 32), id_dkv, (i > 0 || ks > 0) ? 1u : 0u);
              ptx::mma_commit(bar(kGFree));
            }
            __syncwarp();
            if (i + 1 < rows.n) issue_s(tile + 1, i + 1);  // (behind dV, which reads P out of the same columns)
            wait(kDsFull, tile, 72);
            ptx::tc_fence_after_sync();
            if (ptx::elect_one()) {
              for (int ks = 0; ks < keys16; ++ks)  // dQ first: the next dP waits until it has been read out
                ptx::mma_ss_lohi(tmem + kColDp, (uint32_t)ds_mn + (uint32_t)ks * 128, (uint32_t)(ds_mn >> 32),
                                 (uint32_t)k_mn + (uint32_t)ks * 128, (uint32_t)(k_mn >> 32), id_dq, ks > 0);
              ptx::mma_commit(bar(kDqFull));
              for (int ks = 0; ks < r16; ++ks)
                ptx::mma_ss_lohi(tmem + kColDk, (uint32_t)ds_k + (uint32_t)(ks >> 2) * (kChunk >> 4) + (uint32_t)(ks & 3) * 2,
                                 (uint32_t)(ds_k >> 32), (uint32_t)q_mn + so + (uint32_t)ks * 128, (uint32_t)(q_mn >> 32), id_dkv,
                                 (i > 0 || ks > 0) ? 1u : 0u);
              ptx::mma_commit(bar(kQFree + (tile & 1u)));
              if (i + 1 == rows.n) ptx::mma_commit(bar(kAccFull));
            }
            __syncwarp();
          }
        }
      }
    } else {
      // =============================== partial row tiles =========================================
      const int t64 = tid - 14 * 32;
      uint32_t tile = 0;
      auto zero_rows = [&](uint32_t off, int nrow) {  // rows [nrow, 128) of a tile: other tokens' values, whatever they are
#pragma unroll
        for (int c = 0; c < HD / 64; ++c) {
          uint4* const z = reinterpret_cast<uint4*>(smem + off + c * kChunk) + nrow * 8;
          for (int x = t64; x < (kTile - nrow) * 8; x += 64) z[x] = make_uint4(0, 0, 0, 0);
        }
        ptx::fence_proxy_async_smem();
      };
      for (;;) {
        const int idx = next_item();
        if (idx < 0) break;
        const Item it = decode(a, idx);
        for (int kt = 0; kt < it.n_kt; ++kt) {
          const RowList rows = rows_of(a, it, kt);
          for (int i = 0; i < rows.n; ++i, ++tile) {
            // (these warps see every tile, whole ones too: a parity wait must not skip phases)
            const RowTile t = row_tile(a, it, rows, i);
            wait(kQFull + (tile & 1u), tile >> 1, 74);
            if (t.nrow < kTile) {
              zero_rows(L::kOffQ + (tile & 1u) * L::kTileBytes, t.nrow);
              arrive(kQTail + (tile & 1u));
            }
            arrive(kQFree + (tile & 1u));
            wait(kGFull, tile, 75);
            if (t.nrow < kTile) {
              zero_rows(L::kOffG, t.nrow);
              arrive(kGTail);
            }
            arrive(kGFree);
          }
        }
      }
    }
  } else if (warp >= 8) {
    // =============================== outputs =====================================================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 176;");
    const int row = tid & 127;
    const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    uint32_t tile = 0, kts = 0, fills = 0;
    // 32 rows of 128 bytes pass through one of the warp's two 4 KB slabs, so that they leave as whole rows by TMA.  (A thread
    // owns a row: stored directly, one instruction touches 32 lines.)
    const uint32_t slab0 = sbase + L::kOffOut + (uint32_t)(warp & 3) * 8192u;
    auto slab = [&]() { return slab0 + (fills & 1u) * 4096u; };
    auto put = [&](int piece, uint4 w) {
      *reinterpret_cast<uint4*>(smem + (slab() - sbase) + lane * 128 + ((piece ^ (lane & 7)) << 4)) = w;
    };
    auto begin_fill = [&]() {  // the slab's previous transfer has read it
      if (lane == 0) ptx::bulk_wait_read_but_one();
      __syncwarp();
    };
    auto end_fill = [&]() {  // fill visible to the TMA; the caller issues from lane 0
      ptx::fence_proxy_async_smem();
      __syncwarp();
    };
    auto put_f32 = [&](const uint32_t (&x)[32], float f) {  // 32 columns
#pragma unroll
      for (int i = 0; i < 8; ++i)
        put(i, make_uint4(__float_as_uint(__uint_as_float(x[4 * i]) * f), __float_as_uint(__uint_as_float(x[4 * i + 1]) * f),
                          __float_as_uint(__uint_as_float(x[4 * i + 2]) * f), __float_as_uint(__uint_as_float(x[4 * i + 3]) * f)));
    };
    auto pack8 = [&](const uint32_t (&x)[32], int i, float f) {
      return make_uint4(pack_bf16(__uint_as_float(x[i]) * f, __uint_as_float(x[i + 1]) * f),
                        pack_bf16(__uint_as_float(x[i + 2]) * f, __uint_as_float(x[i + 3]) * f),
                        pack_bf16(__uint_as_float(x[i + 4]) * f, __uint_as_float(x[i + 5]) * f),
                        pack_bf16(__uint_as_float(x[i + 6]) * f, __uint_as_float(x[i + 7]) * f));
    };

    // dV, then dK of a key tile: thread = key
    auto drain_acc = [&](const Item& it, int kt) {
      const int j = kt * kTile + row, jw = kt * kTile + (warp & 3) * 32;  // this key, the warp's first
      const int n_list = it.l0 + it.len;
      const int pre_end = a.pre == nullptr ? 0 : it.m == 0 ? it.len : it.l0;  // keys whose sums other items share
      const bool whole = jw >= pre_end && jw + 32 <= n_list;                  // 32 own keys
      const bool mine = j >= pre_end && j < n_list;
#pragma unroll 1
      for (int x = 0; x < 2 * HD; x += 32) {
        const bool is_k = x >= HD;
        const int c0 = x & (HD - 1);
        const float f = is_k ? a.scale : 1.f;
        uint32_t v[32];
        __syncwarp();
        ptx::tmem_ld32(lanes + (is_k ? kColDk : kColDv) + (uint32_t)c0, v);
        ptx::tmem_wait_ld(v);
        if (x + 32 == 2 * HD) {
          ptx::tc_fence_before_sync();
          arrive(kAccFree);
        }
        if (jw < pre_end) {  // (rows beyond the prefix go to rows of the sums that nothing reads)
          begin_fill();
          put_f32(v, f);
          end_fill();
          if (lane == 0) {
            ptx::tma_add_4d(&maps.pre, slab(), c0, ((is_k ? 0 : a.B) + it.b) * a.Nk + it.g, jw, 0);
            ptx::bulk_commit();
          }
          ++fills;
        }
        if (whole) {
          if ((c0 & 32) == 0) begin_fill();
#pragma unroll
          for (int i = 0; i < 32; i += 8) put(((c0 & 32) + i) >> 3, pack8(v, i, f));
          if (c0 & 32) {
            end_fill();
            if (lane == 0) {
              ptx::tma_store_4d(is_k ? &maps.dk : &maps.dv, slab(), c0 - 32, it.g, it.start + jw - it.l0, it.b);
              ptx::bulk_commit();
            }
            ++fills;
          }
        } else if (mine) {
          const View& out = is_k ? a.dk : a.dv;
          __nv_bfloat16* const dst = reinterpret_cast<__nv_bfloat16*>(out.ptr) + (int64_t)it.b * out.sb + (int64_t)it.g * out.sh +
                                     (int64_t)(it.start + j - it.l0) * out.ss + c0;
#pragma unroll
          for (int i = 0; i < 32; i += 8) *reinterpret_cast<uint4*>(dst + i) = pack8(v, i, f);
        }
      }
    };

    for (;;) {
      const int idx = next_item();
      if (idx < 0) break;
      const Item it = decode(a, idx);
      for (int kt = 0; kt < it.n_kt; ++kt, ++kts) {
        const RowList rows = rows_of(a, it, kt);
        for (int i = 0; i < rows.n; ++i, ++tile) {
          // dQ: thread = row
          const RowTile t = row_tile(a, it, rows, i);
          const int row_w = (warp & 3) * 32, tok_w = t.t0 + (row_w >> a.g_shift);  // the warp's first row
          const bool sum32 = a.M > 1 && (!t.own || it.m == a.M - 1);               // rows of the query block
          // own rows: the key tiles that see this row tile are 0 .. last
          const int last = t.own ? (it.l0 + min(it.len, t.t0 + (kTile >> a.g_shift)) - 1) / kTile : 0;
          float4* const part = reinterpret_cast<float4*>(a.part) + ((size_t)blockIdx.x * a.row_tiles + t.r) * (HD / 4) * 128 + row;
          const bool take = !sum32 && kt > 0 && row_w < t.nrow, leave = !sum32 && kt < last;
          float all[HD / 32][32] = {};
          if (take) {  // the partial sum so far: on its way while the product is computed
#pragma unroll
            for (int ch = 0; ch < HD / 32; ++ch)
#pragma unroll
              for (int q = 0; q < 8; ++q) *reinterpret_cast<float4*>(&all[ch][4 * q]) = part[(size_t)(ch * 8 + q) * 128];
          }
          wait(kDqFull, tile, 76);
          ptx::tc_fence_after_sync();
          __syncwarp();
#pragma unroll
          for (int ch = 0; ch < HD / 32; ++ch) {
            uint32_t x[32];
            ptx::tmem_ld32(lanes + kColDp + (uint32_t)ch * 32, x);
            ptx::tmem_wait_ld(x);
#pragma unroll
            for (int q = 0; q < 32; ++q) all[ch][q] += __uint_as_float(x[q]);
          }
          ptx::tc_fence_before_sync();
          arrive(kDqFree);  // out of tensor memory: the next tile's dP may overwrite it
          if (row_w >= t.nrow) continue;
          const float f = a.scale;
#pragma unroll
          for (int ch = 0; ch < HD / 32; ++ch) {
            uint32_t (&v)[32] = *reinterpret_cast<uint32_t (*)[32]>(&all[ch]);
            if (sum32) {  // (rows beyond the block go to rows of the sums that nothing reads)
              begin_fill();
              put_f32(v, f);
              end_fill();
              if (lane == 0) {
                ptx::tma_add_4d(&maps.dq32, slab(), ch * 32, it.g * a.G, tok_w, it.b);
                ptx::bulk_commit();
              }
              ++fills;
              continue;
            }
            if (leave) {
#pragma unroll
              for (int q = 0; q < 8; ++q)
                part[(size_t)(ch * 8 + q) * 128] = make_float4(__uint_as_float(v[4 * q]), __uint_as_float(v[4 * q + 1]),
                                                               __uint_as_float(v[4 * q + 2]), __uint_as_float(v[4 * q + 3]));
            } else if (row_w + 32 <= t.nrow) {
              if ((ch & 1) == 0) begin_fill();
#pragma unroll
              for (int q = 0; q < 32; q += 8) put((ch & 1) * 4 + (q >> 3), pack8(v, q, f));
              if (ch & 1) {
                end_fill();
                if (lane == 0) {
                  ptx::tma_store_4d(&maps.dq, slab(), (ch - 1) * 32, it.g * a.G, it.start + tok_w, it.b);
                  ptx::bulk_commit();
                }
                ++fills;
              }
            } else if (row < t.nrow) {
              __nv_bfloat16* const dst = reinterpret_cast<__nv_bfloat16*>(a.dq.ptr) + (int64_t)it.b * a.dq.sb +
                                         (int64_t)(it.g * a.G + (row & (a.G - 1))) * a.dq.sh +
                                         (int64_t)(t.slot + (row >> a.g_shift)) * a.dq.ss + ch * 32;
#pragma unroll
              for (int q = 0; q < 32; q += 8) *reinterpret_cast<uint4*>(dst + q) = pack8(v, q, f);
            }
          }
        }
        wait(kAccFull, kts, 77);
        ptx::tc_fence_after_sync();
        drain_acc(it, kt);
      }
    }
    if (lane == 0) ptx::bulk_wait();
  } else {
    // =============================== element-wise part ===========================================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 136;");
    const int wg = warp >> 2, row = tid & 127;
    const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)wg * 64;
    uint8_t* const ds_row = smem + L::kOffDs + wg * kChunk + row * 128;
    uint32_t tile = 0, kts = 0;
    // one of K / V of list positions [128 kt, 128 kt + 128) -> shared memory
    auto load = [&](const View& x, uint32_t to, const Item& it, int kt) {
      constexpr int kPieces = HD / 8, kStep = 256 / kPieces;
      const int c = tid % kPieces;
      const __nv_bfloat16* const base = reinterpret_cast<const __nv_bfloat16*>(x.ptr) + (int64_t)it.b * x.sb + (int64_t)it.g * x.sh + c * 8;
#pragma unroll
      for (int r0 = 0; r0 < kTile; r0 += kStep) {
        const int r = r0 + tid / kPieces, j = kt * kTile + r;
        const bool ok = j < it.l0 + it.len;
        const int slot = !ok ? it.start : j < it.l0 ? it.s0 + j : it.start + j - it.l0;
        cp_async16_zfill(smem + to + (uint32_t)(c >> 3) * kChunk + (uint32_t)r * 128u + (uint32_t)(((c & 7) ^ (r & 7)) << 4),
                         base + (int64_t)slot * x.ss, ok);
      }
      cp_async_commit();
    };
    for (;;) {
      const int idx = next_item();
      if (idx < 0) break;
      const Item it = decode(a, idx);
      for (int kt = 0; kt < it.n_kt; ++kt, ++kts) {
        load(a.v, L::kOffV, it, kt);  // (the last dP of the previous key tile is complete: its dS has been computed)
        if (kts > 0) wait(kAccFull, kts - 1, 73);  // every product of the previous key tile is complete
        load(a.k, L::kOffK, it, kt);
        cp_async_wait<0>();
        ptx::fence_proxy_async_smem();
        arrive(kKvFull);
        const RowList rows = rows_of(a, it, kt);
        const int j = kt * kTile + row;  // this thread's key: list position
        for (int i = 0; i < rows.n; ++i, ++tile) {
          const RowTile t = row_tile(a, it, rows, i);
          const uint32_t st = tile & 1u;
          const float* const col = reinterpret_cast<const float*>(smem + L::kOffCol) + st * 2 * kTile + wg * 64;
          // Row-tile columns below cmin do not see this key: causality inside the block; the prefix is not the query
          // rows' business here; positions beyond the list are no keys.
          int cmin = t.own ? (j - it.l0 - t.t0) * a.G : (j < it.l0 ? kTile : 0);
          if (j >= it.l0 + it.len) cmin = kTile;
          cmin -= wg * 64;
          wait(kQFull + st, tile >> 1, 78);
          wait(kSFull, tile, 79);
          ptx::tc_fence_after_sync();
          __syncwarp();
          float p[64];
          {
            uint32_t s[64];
            ptx::tmem_ld32(lanes + kColS, *reinterpret_cast<uint32_t (*)[32]>(&s[0]));
            ptx::tmem_ld32(lanes + kColS + 32, *reinterpret_cast<uint32_t (*)[32]>(&s[32]));
            ptx::tmem_wait_ld(s);
#pragma unroll
            for (int c = 0; c < 64; c += 4) {
              const float4 nl = *reinterpret_cast<const float4*>(col + c);
              p[c] = ptx::ex2(fmaf(__uint_as_float(s[c]), a.scale_log2, nl.x));
              p[c + 1] = ptx::ex2(fmaf(__uint_as_float(s[c + 1]), a.scale_log2, nl.y));
              p[c + 2] = ptx::ex2(fmaf(__uint_as_float(s[c + 2]), a.scale_log2, nl.z));
              p[c + 3] = ptx::ex2(fmaf(__uint_as_float(s[c + 3]), a.scale_log2, nl.w));
            }
          }
          if (__any_sync(0xffffffffu, cmin > 0)) {
#pragma unroll
            for (int c = 0; c < 64; ++c) p[c] = c < cmin ? 0.f : p[c];
          }
          {
            uint32_t pk[32];
#pragma unroll
            for (int c = 0; c < 32; ++c) pk[c] = pack_bf16(p[2 * c], p[2 * c + 1]);
            ptx::tmem_st32(lanes + kColS, pk);
            ptx::tmem_wait_st();
          }
          ptx::tc_fence_before_sync();
          arrive(kPFull);

          wait(kDpFull, tile, 80);  // (dP follows the reading of dQ, so every product that reads dS is complete too)
          ptx::tc_fence_after_sync();
          __syncwarp();
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t x[32];
            ptx::tmem_ld32(lanes + kColDp + (uint32_t)h * 32, x);
            ptx::tmem_wait_ld(x);
#pragma unroll
            for (int c = 0; c < 32; c += 8) {
              const float4 d0 = *reinterpret_cast<const float4*>(col + kTile + h * 32 + c);
              const float4 d1 = *reinterpret_cast<const float4*>(col + kTile + h * 32 + c + 4);
              const float* pp = &p[h * 32 + c];
              uint4 w;
              w.x = pack_bf16(pp[0] * (__uint_as_float(x[c]) - d0.x), pp[1] * (__uint_as_float(x[c + 1]) - d0.y));
              w.y = pack_bf16(pp[2] * (__uint_as_float(x[c + 2]) - d0.z), pp[3] * (__uint_as_float(x[c + 3]) - d0.w));
              w.z = pack_bf16(pp[4] * (__uint_as_float(x[c + 4]) - d1.x), pp[5] * (__uint_as_float(x[c + 5]) - d1.y));
              w.w = pack_bf16(pp[6] * (__uint_as_float(x[c + 6]) - d1.z), pp[7] * (__uint_as_float(x[c + 7]) - d1.w));
              *reinterpret_cast<uint4*>(ds_row + (((h * 4 + (c >> 3)) ^ (row & 7)) << 4)) = w;
            }
          }
          ptx::fence_proxy_async_smem();
          ptx::tc_fence_before_sync();
          arrive(kDsFull);
        }
      }
    }
  }
  ptx::tc_fence_before_sync();
  ptx::end_of_waits(waits, [](int mark) { return mark; }, a.status);
  if (warp == 0) ptx::tmem_dealloc(tmem, 512);
}

__device__ __forceinline__ bool slot_in_block(const BwdTcArgs& a, int b, int s) {
  int lo = 0, hi = a.M;  // first block that starts behind s (blk_start is non-decreasing)
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (a.blk_start[(size_t)b * a.M + mid] <= s) lo = mid + 1; else hi = mid;
  }
  if (lo == 0) return false;
  int start, len;
  span_of(a, b, lo - 1, start, len);
  return s < start + len;
}

// delta = rowsum(dO * O): eight slots and all heads of a prompt per CTA, one token per warp, so that a warp's reads are
// contiguous; the sums change places in shared memory, because delta is kept by head.  The same warps write the zeros of
// the slots outside every block; all threads clear the accumulators and the item counter.  Bound by memory: reads O and
// dO once.  The first block orders the items.  (By warps that owned 32 slots of one head, reads 8 KB apart, a grid of 100
// documents of 32..256 tokens took 72 us, now 62; 16 slots per CTA: 70.)
constexpr int kPrepTok = 8;
template <int HD>
__global__ void __launch_bounds__(256, 4) attn_bwd_tc_prep_kernel(BwdTcArgs a, float4* zero, int64_t n_zero) {
  if (a.order && blockIdx.x == 0) {
    // (prompt, block) pairs by length, longest first (counting sort, one bucket per 8 tokens up to 512)
    __shared__ int first[64];
    const int n = a.B * a.M;
    auto bucket = [&](int i) {
      int start, len;
      span_of(a, i / a.M, i % a.M, start, len);
      return 63 - min(63, (len + 7) >> 3);
    };
    if (threadIdx.x < 64) first[threadIdx.x] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += 256) atomicAdd(&first[bucket(i)], 1);
    __syncthreads();
    if (threadIdx.x == 0) {
      int sum = 0;
      for (int i = 0; i < 64; ++i) {
        const int c = first[i];
        first[i] = sum;
        sum += c;
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += 256) a.order[atomicAdd(&first[bucket(i)], 1)] = i;
    return;
  }
  const int skip = a.order ? 1 : 0, blk = blockIdx.x - skip;
  const int64_t gid = (int64_t)blk * 256 + threadIdx.x;
  for (int64_t i = gid; i < n_zero; i += (int64_t)(gridDim.x - skip) * 256) zero[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (gid == 0) *a.counter = 0;
  constexpr int kLanes = HD / 8, kRows = 32 / kLanes;  // lanes per row, heads per access of a warp
  constexpr int kHeads = 64;                            // heads per pass through shared memory
  __shared__ float s_delta[kHeads][kPrepTok + 1];
  __shared__ unsigned s_live;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int groups = (a.S + kPrepTok - 1) / kPrepTok;
  const int b = blk / groups, t0 = (blk % groups) * kPrepTok;
  if (warp == 0) {
    const unsigned l = __ballot_sync(0xffffffffu, lane < kPrepTok && t0 + lane < a.S && slot_in_block(a, b, t0 + lane));
    if (lane == 0) s_live = l;
  }
  __syncthreads();
  const unsigned live = s_live;
  const int sub = lane / kLanes, c = (lane % kLanes) * 8;
  auto at = [&](const View& t, int s, int n) {
    return reinterpret_cast<__nv_bfloat16*>(t.ptr) + (int64_t)b * t.sb + (int64_t)s * t.ss + (int64_t)n * t.sh + c;
  };
  auto clear = [&](const View& t, int s, int heads) {
    for (int n = sub; n < heads; n += kRows) *reinterpret_cast<uint4*>(at(t, s, n)) = make_uint4(0, 0, 0, 0);
  };
  for (int n0 = 0; n0 < a.N; n0 += kHeads) {
    const int nh = min(kHeads, a.N - n0);
    for (int t = warp; t < kPrepTok; t += 8) {
      const int s = t0 + t;
      if (!((live >> t) & 1u)) {  // (not read)
        if (s < a.S && n0 == 0) {
          clear(a.dq, s, a.N);
          clear(a.dk, s, a.Nk);
          clear(a.dv, s, a.Nk);
        }
        for (int n = lane; n < nh; n += 32) s_delta[n][t] = 0.f;
        continue;
      }
      const __nv_bfloat16 *const gp = at(a.d_o, s, n0 + sub), *const op = at(a.o, s, n0 + sub);
#pragma unroll 1
      for (int n1 = 0; n1 < nh; n1 += 4 * kRows) {
        uint4 x[4], y[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int n = min(n1 + i * kRows, nh - 1 - sub);  // (past the last head: read again, not kept)
          x[i] = *reinterpret_cast<const uint4*>(gp + (int64_t)n * a.d_o.sh);
          y[i] = *reinterpret_cast<const uint4*>(op + (int64_t)n * a.o.sh);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float d = 0.f;
          auto dot = [&](uint32_t u, uint32_t v) {
            const float2 p = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&u));
            const float2 q = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&v));
            d = fmaf(p.y, q.y, fmaf(p.x, q.x, d));
          };
          dot(x[i].x, y[i].x); dot(x[i].y, y[i].y); dot(x[i].z, y[i].z); dot(x[i].w, y[i].w);
#pragma unroll
          for (int off = kLanes / 2; off > 0; off >>= 1) d += __shfl_xor_sync(0xffffffffu, d, off);
          if (c == 0 && n1 + i * kRows + sub < nh) s_delta[n1 + i * kRows + sub][t] = d;
        }
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nh * kPrepTok; i += 256) {
      const int n = i / kPrepTok, t = i % kPrepTok;
      if (t0 + t < a.S) a.delta[((size_t)b * a.N + n0 + n) * a.S + t0 + t] = s_delta[n][t];
    }
    __syncthreads();
  }
}

// fp32 sums -> bf16: dQ of the last block's rows, dK and dV of the prefix.  One thread per 8 elements.
template <int HD>
__global__ void __launch_bounds__(256) attn_bwd_tc_finish_kernel(BwdTcArgs a) {
  const int64_t nq = (int64_t)a.B * a.N * a.max_block_len * (HD / 8), np = a.pre ? (int64_t)a.B * a.Nk * a.max_block_len * (HD / 8) : 0;
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < nq + 2 * np; i += (int64_t)gridDim.x * 256) {
    const bool q = i < nq;
    const int64_t x = q ? i : (i - nq) % np;
    const bool dv = !q && i - nq >= np;
    const int heads = q ? a.N : a.Nk;
    const int c = (int)(x % (HD / 8)) * 8, tok = (int)(x / (HD / 8) % a.max_block_len);
    const int64_t bh = x / ((int64_t)(HD / 8) * a.max_block_len);
    const int h = (int)(bh % heads), b = (int)(bh / heads);
    int start, len;
    span_of(a, b, q ? a.M - 1 : 0, start, len);
    if (tok >= len) continue;
    float v[8];
    load8((q ? a.dq32 : a.pre + (dv ? np * 8 : 0)) + x * 8, v);
    const View& t = q ? a.dq : dv ? a.dv : a.dk;
    store8(reinterpret_cast<__nv_bfloat16*>(t.ptr) + (int64_t)b * t.sb + (int64_t)h * t.sh + (int64_t)(start + tok) * t.ss + c, v);
  }
}

int row_tiles(const brk_attn_bwd_params& p) { return (int)(((int64_t)p.max_block_len * (p.N / p.Nk) + kTile - 1) / kTile); }
// Rows whose keys can span several key tiles need the fp32 dQ scratch.
bool needs_part(const brk_attn_bwd_params& p) { return (int64_t)(p.M > 2 ? 2 : 1) * p.max_block_len > kTile; }
size_t part_bytes(const brk_attn_bwd_params& p) {
  return needs_part(p) ? (size_t)std::max(1, sm_count()) * row_tiles(p) * kTile * p.D * sizeof(float) : 0;
}

template <int HD>
int launch(const brk_attn_bwd_params& p, BwdTcArgs a, float4* zero, int64_t n_zero, cudaStream_t st) {
  const int tok = kTile / a.G, tok_w = std::max(1, 32 / a.G);
  Maps t;
  auto map = [&](CUtensorMap& m, const brk_view& v, int heads, int box_h, int box_s) {
    return make_tmap_bf16(&m, v.ptr, HD, heads, p.S, p.B, v.stride_h, v.stride_s, v.stride_b, box_h, box_s);
  };
  int rc;
  if ((rc = map(t.q, p.q, p.N, a.G, tok)) || (rc = map(t.g, p.d_o, p.N, a.G, tok)) || (rc = map(t.dq, p.dq, p.N, a.G, tok_w)) ||
      (rc = map(t.dk, p.dk, p.Nk, 1, 32)) || (rc = map(t.dv, p.dv, p.Nk, 1, 32)))
    return rc;
  const int64_t mbl = p.max_block_len;
  if ((rc = make_tmap_f32(&t.dq32, a.dq32, HD, p.N, p.max_block_len, p.B, mbl * HD, HD, (int64_t)p.N * mbl * HD, a.G, tok_w))) return rc;
  t.pre = t.dq32;
  if (a.pre && (rc = make_tmap_f32(&t.pre, a.pre, HD, 2 * p.B * p.Nk, p.max_block_len, 1, mbl * HD, HD, 0, 1, 32))) return rc;
  const unsigned prep = (unsigned)p.B * ((p.S + kPrepTok - 1) / kPrepTok) + (a.order ? 1 : 0);
  attn_bwd_tc_prep_kernel<HD><<<prep, 256, 0, st>>>(a, zero, n_zero);
  BRK_LAUNCHED();
  BRK_CUDA(cudaFuncSetAttribute(attn_bwd_tc_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Geo<HD>::kSmem));
  const int sms = sm_count();
  BRK_REQUIRE(sms > 0, BRK_E_CUDA, "could not read the SM count");
  attn_bwd_tc_kernel<HD><<<std::min(sms, a.total_items), kThreads, Geo<HD>::kSmem, st>>>(t, a);
  BRK_LAUNCHED();
  if (p.M > 1) {
    const int64_t n = (int64_t)p.B * (p.N + (a.pre ? 2 * p.Nk : 0)) * p.max_block_len * (HD / 8);
    attn_bwd_tc_finish_kernel<HD><<<(unsigned)std::min<int64_t>((n + 255) / 256, sms * 8), 256, 0, st>>>(a);
    BRK_LAUNCHED();
  }
  return BRK_OK;
}

}  // namespace

// bf16 with a group size that divides a row tile, and blocks short enough for the dQ scratch of a CTA (512 tokens at four
// heads per KV head).  Longer blocks go to the warp-level kernels, which split a block over CTAs.
bool attn_bwd_tc_supported(const brk_attn_bwd_params& p) {
  const int G = p.Nk > 0 ? p.N / p.Nk : 0;
  return p.dtype == BRK_BF16 && (p.D == 64 || p.D == 128) && (G == 1 || G == 2 || G == 4 || G == 8) && row_tiles(p) <= kMaxRowTiles;
}
// item counter and item order, then the dQ scratch
static size_t head_bytes(const brk_attn_bwd_params& p) { return (256 + (size_t)p.B * p.M * sizeof(int) + 255) & ~(size_t)255; }
size_t attn_bwd_tc_extra_bytes(const brk_attn_bwd_params& p) { return p.M > 2 || part_bytes(p) > 0 ? head_bytes(p) + part_bytes(p) : 0; }

// ws32: the prefix sums, right in front of dq32 (two blocks or fewer: accumulators of which only the item counter is used);
// extra: the bytes of attn_bwd_tc_extra_bytes
int attn_bwd_tc_launch(const brk_attn_bwd_params& p, float* delta, float* ws32, float* dq32, void* extra, int32_t* status,
                       cudaStream_t st) {
  BwdTcArgs a{};
  a.q = make_view(p.q); a.k = make_view(p.k); a.v = make_view(p.v); a.o = make_view(p.o); a.d_o = make_view(p.d_o);
  a.dq = make_view(p.dq); a.dk = make_view(p.dk); a.dv = make_view(p.dv);
  a.lse = p.lse;
  a.delta = delta;
  a.blk_start = p.blk_start; a.blk_len = p.blk_len;
  a.status = status;
  a.B = p.B; a.N = p.N; a.Nk = p.Nk; a.S = p.S; a.M = p.M; a.G = p.N / p.Nk; a.max_block_len = p.max_block_len;
  while ((1 << a.g_shift) < a.G) ++a.g_shift;
  a.row_tiles = row_tiles(p);
  BRK_REQUIRE((int64_t)p.B * p.Nk * p.M < (1ll << 31), BRK_E_UNSUPPORTED, "too many work items");
  a.total_items = p.B * p.Nk * p.M;
  a.scale = p.scale;
  a.scale_log2 = p.scale * 1.4426950408889634f;
  // With two blocks or fewer no document adds to the prefix's dK / dV: block 0's own item stores them.
  const int64_t n_pre = p.M > 2 ? 2ll * p.B * p.Nk * p.max_block_len * p.D : 0, n_q = p.M > 1 ? (int64_t)p.B * p.N * p.max_block_len * p.D : 0;
  // The prefix sums sit directly in front of dq32: one range to clear.
  a.pre = n_pre ? dq32 - n_pre : nullptr;
  a.dq32 = dq32;
  unsigned char* const x = static_cast<unsigned char*>(extra);
  const bool has_extra = attn_bwd_tc_extra_bytes(p) > 0;
  a.counter = has_extra ? reinterpret_cast<int*>(x) : reinterpret_cast<int*>(ws32);
  a.order = has_extra && p.M > 2 ? reinterpret_cast<int*>(x + 256) : nullptr;
  a.part = part_bytes(p) ? reinterpret_cast<float*>(x + head_bytes(p)) : nullptr;
  float4* const zero = reinterpret_cast<float4*>(dq32 - n_pre);
  return p.D == 128 ? launch<128>(p, a, zero, (n_pre + n_q) / 4, st) : launch<64>(p, a, zero, (n_pre + n_q) / 4, st);
}

}  // namespace brk
