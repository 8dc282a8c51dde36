// Raw logits of the last R slots of a prompt against every slot (the registered attention function's second return
// value) and the gradient of those logits.
//
//   raw_scores_mma_kernel   bf16: out[row, s] = round(q[row] * scale) . k[s], masked.  The G*R rows of a KV head share
//                           one read of every key; a CTA keeps 16 rows per warp as MMA A fragments and walks through
//                           64-key tiles (cp.async, two buffers).
//   raw_scores_f32_kernel   fp32: 64 rows x 64 keys per CTA, 4 x 4 products per thread on CUDA cores.
//   raw_bwd_mma_kernel / raw_bwd_f32_kernel
//                           dk[s] (+)= scale * sum over rows of d_raw[row, s] q[row], and
//                           dq[row] (+)= scale * sum over slots of d_raw[row, s] k[s].  One pass over d_raw and k: a
//                           CTA owns 64-slot tiles, stores dk itself and adds its share of dq into an fp32 scratch
//                           that raw_bwd_rows_kernel puts into the last R rows.
//
// All four are bound by memory: per prompt of 100 documents (32/8 heads, 16 rows, 16,320 slots) the forward moves
// 33 MB of keys and writes 17 MB of logits, the backward reads those and updates 33 MB of dk, for 2 and 4 GFLOP.
// Measured there: forward 18.6 us (one thread per key row on CUDA cores: 230 us); 4 prompts of 20 documents (14,080
// slots): forward 17 us (195), backward 29 us (fp32 matrix products, casts, fills and sums in PyTorch: about 500);
// fp32 forward, 1 prompt of 20 documents: 21 us (81).
#include <algorithm>

#include "brk_common.cuh"
#include "mma_bf16.cuh"
#include "score_args.cuh"
#include "tc_ptx.cuh"

namespace brk {
namespace {

constexpr int kThreads = 128;      // bf16 kernels: four warps
constexpr int kThreadsF = 256;     // fp32 kernels
constexpr int kKeys = 64;          // slots per tile
constexpr int kRowsPass = 64;      // (head, row) pairs per pass: four warps of 16
constexpr int kMaxSharedSpans = 1024;  // block spans are searched in shared memory up to this many blocks

// block index of a slot, or -1 for padding (bs is non-decreasing)
__device__ __forceinline__ int block_of(const int32_t* bs, const int32_t* bl, int M, int s) {
  int lo = 0, hi = M;  // first index with bs > s
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (bs[mid] <= s) lo = mid + 1; else hi = mid;
  }
  const int m = lo - 1;
  return (m >= 0 && s < bs[m] + bl[m]) ? m : -1;
}

// is the pair (query slot qslot of block qb, key slot s of block kblk) visible?
__device__ __forceinline__ bool pair_ok(int qb, int qslot, int kblk, int s, int M) {
  return qb >= 0 && kblk >= 0 &&
         ((kblk == qb && s <= qslot) || (qb == M - 1 && kblk < qb) || (qb > 0 && qb < M - 1 && kblk == 0));
}

// The 16-byte pieces of a staged key row are permuted by the row so that both kinds of eight-row groups the MMA
// fragments are read in (rows 8i + {0,1} + 2t, i = 0..3, here; eight consecutive rows in the backward) fall on
// eight different bank groups.
__device__ __forceinline__ int swz(int row, int piece) { return piece ^ ((((row >> 3) & 3) << 1 | (row & 1)) & 7); }

// Bound by instruction issue (64 x 64 logits per tile, each with its visibility).  Nearly every tile lies in front of the
// query block that holds all R rows: there a key is visible if it exists, so a thread's eight keys take eight bits of a
// ballot, and where the prompt has no padding nothing is looked up at all.  (With every pair tested on its own a prompt of 100
// documents took 22 us, 1,150 instructions per warp and tile; now 18.6.)
template <int D>
constexpr int kRawPerSm = D == 128 ? 4 : 5;  // CTAs per SM
template <int D>
__global__ void __launch_bounds__(kThreads, kRawPerSm<D>) raw_scores_mma_kernel(ScoreArgs a, __nv_bfloat16* __restrict__ out, float neg,
                                                                              int wide) {
  constexpr int kPieces = D / 8;
  __shared__ __align__(16) __nv_bfloat16 ktile[2][kKeys][D];
  __shared__ int s_kblk[2][kKeys];
  __shared__ int s_qblk[64];
  __shared__ unsigned s_bits[2][kKeys / 32];  // which keys of the tile exist
  __shared__ int s_sum[kThreads / 32];
  extern __shared__ int32_t s_spans[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, tq = lane & 3;
  const int G = a.N / a.Nk, GR = G * a.R;
  const int b = blockIdx.y / a.Nk, g = blockIdx.y % a.Nk;
  const int32_t* bs = a.blk_start + (size_t)b * a.M;
  const int32_t* bl = a.blk_len + (size_t)b * a.M;
  ptx::grid_dependency_wait();  // (launched beside the end of the attention call's last kernel: 156.6 -> 154.2 us for both)
  int sum = 0;  // keys in front of the last block
  for (int i = tid; i < a.M; i += kThreads) {
    const int start = bs[i], len = bl[i];
    if (i < a.M - 1) sum += len;
    if (a.M <= kMaxSharedSpans) {
      s_spans[i] = start;
      s_spans[a.M + i] = len;
    }
  }
  sum = __reduce_add_sync(0xffffffffu, sum);
  if (lane == 0) s_sum[warp] = sum;
  __syncthreads();
  if (a.M <= kMaxSharedSpans) {
    bs = s_spans;
    bl = s_spans + a.M;
  }
  const int first = bs[0], own = bs[a.M - 1];
  const bool all_query = a.S - a.R >= own && a.S <= own + bl[a.M - 1];  // all R rows belong to the last block
  const bool no_gaps = s_sum[0] + s_sum[1] + s_sum[2] + s_sum[3] == own - first;
  auto in_front = [&](int tile) { return all_query && (tile + 1) * kKeys <= own; };           // visible: every key that exists
  auto solid = [&](int tile) { return no_gaps && in_front(tile) && tile * kKeys >= first; };  // every key exists
  if (tid < a.R) s_qblk[tid] = block_of(bs, bl, a.M, a.S - a.R + tid);
  const int n_tiles = (a.S + kKeys - 1) / kKeys;
  const __nv_bfloat16* kb = reinterpret_cast<const __nv_bfloat16*>(a.k.ptr) + (int64_t)b * a.k.sb + (int64_t)g * a.k.sh;
  const int row0 = tid / kPieces, pc = tid % kPieces;
  constexpr int kRowStep = kThreads / kPieces;
  const int64_t step = kRowStep * a.k.ss;
  auto request = [&](int tile, int buf) {
    const __nv_bfloat16* src = kb + (int64_t)(tile * kKeys + row0) * a.k.ss + pc * 8;
    if ((tile + 1) * kKeys <= a.S) {
#pragma unroll
      for (int j = 0; j < kKeys / kRowStep; ++j, src += step)
        cp_async16(&ktile[buf][row0 + j * kRowStep][swz(row0 + j * kRowStep, pc) * 8], src);
    } else {
#pragma unroll 1
      for (int row = row0; row < kKeys; row += kRowStep, src += step) {
        const bool ok = tile * kKeys + row < a.S;
        cp_async16_zfill(&ktile[buf][row][swz(row, pc) * 8], ok ? src : kb, ok);
      }
    }
    if (tid < kKeys && !solid(tile)) {
      const int s = tile * kKeys + tid, kblk = s < a.S ? block_of(bs, bl, a.M, s) : -1;
      s_kblk[buf][tid] = kblk;
      const unsigned bits = __ballot_sync(0xffffffffu, kblk >= 0);
      if (lane == 0) s_bits[buf][warp] = bits;
    }
  };
  for (int r0 = 0; r0 < GR; r0 += kRowsPass) {
    // Warps split the pass's rows 16 by 16; with 32 rows or fewer the spare warps take the other half of the keys.
    const int groups = min(kRowsPass, GR - r0) > 32 ? 4 : (min(kRowsPass, GR - r0) > 16 ? 2 : 1);
    const int rg = warp % groups, half = warp / groups;
    const int c_lo = groups == 4 ? 0 : half * 32, c_hi = groups == 4 ? kKeys : (half < 2 ? c_lo + 32 : c_lo);
    __syncthreads();  // the previous pass has read both buffers
    int tile = blockIdx.x, buf = 0;
    if (tile < n_tiles) request(tile, 0);
    cp_async_commit();
    uint32_t qa[D / 16][4];  // rows r0 + 16 rg + {gq, gq + 8}, scaled and rounded as the reference's Q * scaling
    const int rows[2] = {r0 + rg * 16 + gq, r0 + rg * 16 + gq + 8};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int row = min(rows[h], GR - 1);
      const __nv_bfloat16* qp = reinterpret_cast<const __nv_bfloat16*>(a.q.ptr) + (int64_t)b * a.q.sb +
                                (int64_t)(g * G + row / a.R) * a.q.sh + (int64_t)(a.S - a.R + row % a.R) * a.q.ss;
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks)
#pragma unroll
        for (int w = 0; w < 2; ++w) {
          const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(qp + ks * 16 + w * 8 + 2 * tq));
          qa[ks][h + 2 * w] = pack_bf16(x.x * a.scale, x.y * a.scale);
        }
    }
    int64_t orow[2];
    int qb[2], qslot[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int row = min(rows[h], GR - 1);
      orow[h] = (((int64_t)b * a.N + g * G + row / a.R) * a.R + row % a.R) * a.S;
      qslot[h] = a.S - a.R + row % a.R;
      qb[h] = s_qblk[row % a.R];
    }
    for (; tile < n_tiles; tile += gridDim.x, buf ^= 1) {
      if (tile + (int)gridDim.x < n_tiles) request(tile + gridDim.x, buf ^ 1);
      cp_async_commit();
      cp_async_wait<1>();
      __syncthreads();
      for (int c0 = c_lo; c0 < c_hi; c0 += 32) {
        // Column n of product t belongs to key c0 + 8 (n / 2) + 2 t + n % 2, so that a thread's results of the four
        // products are eight consecutive keys: one 16-byte store.
        float c[4][4];
#pragma unroll
        for (int t = 0; t < 4; ++t) c[t][0] = c[t][1] = c[t][2] = c[t][3] = 0.f;
        const int mi = lane >> 3, r8 = lane & 7;
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
#pragma unroll
          for (int tp = 0; tp < 2; ++tp) {
            uint32_t f[4];
            const int key = c0 + 8 * (r8 >> 1) + 2 * (2 * tp + (mi >> 1)) + (r8 & 1);
            ldsm_x4(f, &ktile[buf][key][swz(key, 2 * ks + (mi & 1)) * 8]);
            mma16816(c[2 * tp], qa[ks], f[0], f[1]);
            mma16816(c[2 * tp + 1], qa[ks], f[2], f[3]);
          }
        }
        const int s0 = tile * kKeys + c0 + 8 * tq;
        if (s0 >= a.S) continue;
        const bool front = in_front(tile);
        const unsigned exist = solid(tile) ? 0xffu : (s_bits[buf][c0 >> 5] >> (8 * tq)) & 0xffu;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (rows[h] >= GR) continue;
          float v[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] = c[i >> 1][2 * h + (i & 1)];
          if (!front) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
              if (!pair_ok(qb[h], qslot[h], s_kblk[buf][c0 + 8 * tq + i], s0 + i, a.M)) v[i] = neg;
          } else if (exist != 0xffu) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
              if (!((exist >> i) & 1u)) v[i] = neg;
          }
          __nv_bfloat16* o = out + orow[h] + s0;
          if (wide) {
            store8(o, v);
          } else {
#pragma unroll
            for (int i = 0; i < 8; ++i)
              if (s0 + i < a.S) o[i] = __float2bfloat16_rn(v[i]);
          }
        }
      }
      __syncthreads();  // the buffer is refilled by the next iteration's copy
    }
  }
}

// 64 (head, row) pairs x 64 keys per CTA; thread (ty, tx) owns rows ty + 16 i and keys tx + 16 i (rows padded by 16
// bytes: the eight threads of a shared-memory phase read eight different bank groups).
template <int D>
__global__ void __launch_bounds__(kThreadsF) raw_scores_f32_kernel(ScoreArgs a, float* __restrict__ out, float neg) {
  constexpr int kPitch = D + 4;
  extern __shared__ __align__(16) float fsm[];
  float* qs = fsm;                  // [64][kPitch]
  float* ks = fsm + 64 * kPitch;    // [64][kPitch]
  __shared__ int s_kblk[kKeys], s_qblk[64];
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const int G = a.N / a.Nk, GR = G * a.R;
  const int b = blockIdx.y / a.Nk, g = blockIdx.y % a.Nk, s0 = blockIdx.x * kKeys;
  const int32_t* bs = a.blk_start + (size_t)b * a.M;
  const int32_t* bl = a.blk_len + (size_t)b * a.M;
  if (tid < a.R) s_qblk[tid] = block_of(bs, bl, a.M, a.S - a.R + tid);
  if (tid >= 64 && tid < 64 + kKeys) s_kblk[tid - 64] = s0 + tid - 64 < a.S ? block_of(bs, bl, a.M, s0 + tid - 64) : -1;
  const float* kb = reinterpret_cast<const float*>(a.k.ptr) + (int64_t)b * a.k.sb + (int64_t)g * a.k.sh;
  for (int i = tid; i < kKeys * (D / 4); i += kThreadsF) {
    const int row = i / (D / 4), d = i % (D / 4) * 4;
    *reinterpret_cast<float4*>(ks + row * kPitch + d) = load4(kb + (int64_t)min(s0 + row, a.S - 1) * a.k.ss + d);
  }
  for (int r0 = 0; r0 < GR; r0 += 64) {
    __syncthreads();
    for (int i = tid; i < 64 * (D / 4); i += kThreadsF) {
      const int rr = i / (D / 4), d = i % (D / 4) * 4, row = min(r0 + rr, GR - 1);
      const float4 x = load4(reinterpret_cast<const float*>(a.q.ptr) + (int64_t)b * a.q.sb +
                             (int64_t)(g * G + row / a.R) * a.q.sh + (int64_t)(a.S - a.R + row % a.R) * a.q.ss + d);
      *reinterpret_cast<float4*>(qs + rr * kPitch + d) = make_float4(x.x * a.scale, x.y * a.scale, x.z * a.scale, x.w * a.scale);
    }
    __syncthreads();
    float acc[4][4] = {};
#pragma unroll 4
    for (int d = 0; d < D; d += 4) {
      float4 q[4], k[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        q[i] = *reinterpret_cast<const float4*>(qs + (ty + 16 * i) * kPitch + d);
        k[i] = *reinterpret_cast<const float4*>(ks + (tx + 16 * i) * kPitch + d);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          acc[i][j] = fmaf(q[i].w, k[j].w, fmaf(q[i].z, k[j].z, fmaf(q[i].y, k[j].y, fmaf(q[i].x, k[j].x, acc[i][j]))));
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = r0 + ty + 16 * i;
      if (row >= GR) continue;
      float* o = out + (((int64_t)b * a.N + g * G + row / a.R) * a.R + row % a.R) * a.S;
      const int qb = s_qblk[row % a.R], qslot = a.S - a.R + row % a.R;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int s = s0 + tx + 16 * j;
        if (s < a.S) o[s] = pair_ok(qb, qslot, s_kblk[tx + 16 * j], s, a.M) ? acc[i][j] : neg;
      }
    }
  }
}

struct RawBwdArgs {
  ScoreArgs s;
  View dq, dk;
  const void* d_raw;  // [B, N, R, S]
  float* dq32;        // [B, N, R, D], zeroed before the launch
  float2* dk32;       // bf16, more than one pass: fp32 sums of dk between the passes, [B, Nk, tile][D / 8][2][thread]
  int add;            // add to dq / dk instead of overwriting
};

// One CTA walks through 64-slot tiles of a (prompt, KV head).  q of 64 (head, row) pairs stays in shared memory; d_raw
// [64 pairs x 64 slots] and k of a tile are staged, dk comes from 16 slots per warp, dq from 16 pairs per warp (held in
// registers over all of the CTA's tiles).  More than 64 pairs: the sums of dk wait in fp32 between the passes, laid out for
// coalesced access by the thread that wrote them, and are rounded once, behind the last (128 pairs, error against 64 bits:
// 1.66e-3, that of the rounding; rounded after every pass it was 2.44e-3).
// d_raw, k and the dk to be added to arrive one tile ahead (two stages, two CTAs per SM): with three CTAs of one stage each,
// 4 prompts of 20 documents took 48 us, most of it waiting for these loads; now 29.
template <int D>
struct RawBwdStage {
  MmaTile<D> k, old;
  MmaTile<kKeys> g;
};
template <int D>
__global__ void __launch_bounds__(kThreads) raw_bwd_mma_kernel(RawBwdArgs a) {
  extern __shared__ __align__(16) unsigned char dyn[];
  MmaTile<D>& qt = *reinterpret_cast<MmaTile<D>*>(dyn);
  RawBwdStage<D>* const stages = reinterpret_cast<RawBwdStage<D>*>(dyn + sizeof(MmaTile<D>));
  const ScoreArgs& s = a.s;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, tq = lane & 3;
  const int G = s.N / s.Nk, GR = G * s.R;
  const int b = blockIdx.y / s.Nk, g = blockIdx.y % s.Nk;
  const int n_tiles = (s.S + kKeys - 1) / kKeys;
  const __nv_bfloat16* kb = reinterpret_cast<const __nv_bfloat16*>(s.k.ptr) + (int64_t)b * s.k.sb + (int64_t)g * s.k.sh;
  __nv_bfloat16* dkb = reinterpret_cast<__nv_bfloat16*>(a.dk.ptr) + (int64_t)b * a.dk.sb + (int64_t)g * a.dk.sh;
  const __nv_bfloat16* gb = reinterpret_cast<const __nv_bfloat16*>(a.d_raw) + (int64_t)(b * s.N + g * G) * s.R * s.S;
  const bool vec = (s.S & 7) == 0;
  for (int r0 = 0; r0 < GR; r0 += kRowsPass) {
    const int nrow = min(kRowsPass, GR - r0);
    __syncthreads();
    for (int i = tid; i < kRowsPass * (D / 8); i += kThreads) {
      const int rr = i / (D / 8), c = i % (D / 8), row = min(r0 + rr, GR - 1);
      cp_async16_zfill(&qt.e[rr][c * 8], reinterpret_cast<const __nv_bfloat16*>(s.q.ptr) + (int64_t)b * s.q.sb +
                           (int64_t)(g * G + row / s.R) * s.q.sh + (int64_t)(s.S - s.R + row % s.R) * s.q.ss + c * 8,
                       rr < nrow);
    }
    float dq[D / 8][4];
#pragma unroll
    for (int i = 0; i < D / 8; ++i) dq[i][0] = dq[i][1] = dq[i][2] = dq[i][3] = 0.f;
    const bool last = r0 + kRowsPass >= GR, add = a.add && last;
    auto request = [&](int tile, RawBwdStage<D>& st) {
      const int s0 = tile * kKeys;
      for (int i = tid; i < kKeys * (D / 8); i += kThreads) {
        const int row = i / (D / 8), c = i % (D / 8), sl = min(s0 + row, s.S - 1);
        cp_async16_zfill(&st.k.e[row][c * 8], kb + (int64_t)sl * s.k.ss + c * 8, s0 + row < s.S);
        if (add) cp_async16_zfill(&st.old.e[row][c * 8], dkb + (int64_t)sl * a.dk.ss + c * 8, s0 + row < s.S);
      }
      if (vec) {
        for (int i = tid; i < kRowsPass * (kKeys / 8); i += kThreads) {
          const int rr = i / (kKeys / 8), c = i % (kKeys / 8) * 8;
          const bool ok = rr < nrow && s0 + c < s.S;
          cp_async16_zfill(&st.g.e[rr][c], gb + (int64_t)(r0 + (ok ? rr : 0)) * s.S + (ok ? s0 + c : 0), ok);
        }
      } else {
        for (int i = tid; i < kRowsPass * kKeys; i += kThreads) {
          const int rr = i / kKeys, c = i % kKeys;
          st.g.e[rr][c] = rr < nrow && s0 + c < s.S ? gb[(int64_t)(r0 + rr) * s.S + s0 + c] : __float2bfloat16_rn(0.f);
        }
      }
    };
    int tile = blockIdx.x, buf = 0;
    if (tile < n_tiles) request(tile, stages[0]);
    cp_async_commit();
    for (; tile < n_tiles; tile += gridDim.x, buf ^= 1) {
      const int s0 = tile * kKeys;
      if (tile + (int)gridDim.x < n_tiles) request(tile + gridDim.x, stages[buf ^ 1]);
      cp_async_commit();
      cp_async_wait<1>();
      __syncthreads();
      MmaTile<D>& kt = stages[buf].k;
      const MmaTile<D>& old = stages[buf].old;
      const MmaTile<kKeys>& gt = stages[buf].g;
      // dq: pairs 16 warp .. + 15, contraction over the 64 slots
#pragma unroll
      for (int c0 = 0; c0 < kKeys; c0 += 16) {
        uint32_t af[4];
        ldsm_x4(af, &gt.e[warp * 16 + (lane & 7) + ((lane >> 3) & 1) * 8][c0 + (lane >> 4) * 8]);
        mm_nn_acc<D>(dq, af, kt, c0, lane);
      }
      // dk: slots 16 warp .. + 15, contraction over the 64 pairs (A = d_raw transposed)
      float dk[D / 8][4];
#pragma unroll
      for (int i = 0; i < D / 8; ++i) dk[i][0] = dk[i][1] = dk[i][2] = dk[i][3] = 0.f;
#pragma unroll
      for (int p0 = 0; p0 < kRowsPass; p0 += 16) {
        uint32_t af[4];
        ldsm_x4_t(af, &gt.e[p0 + (lane & 7) + (lane >> 4) * 8][warp * 16 + ((lane >> 3) & 1) * 8]);
        mm_nn_acc<D>(dk, af, qt, p0, lane);
      }
      if (GR > kRowsPass) {
        float2* const sum = a.dk32 + ((int64_t)blockIdx.y * n_tiles + tile) * (D / 4) * kThreads + tid;
#pragma unroll
        for (int nt = 0; nt < D / 8; ++nt)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float2* const p = sum + (nt * 2 + h) * kThreads;
            if (r0 > 0) {
              const float2 x = *p;
              dk[nt][2 * h] += x.x;
              dk[nt][2 * h + 1] += x.y;
            }
            if (!last) *p = make_float2(dk[nt][2 * h], dk[nt][2 * h + 1]);
          }
        if (!last) {
          __syncthreads();  // the stage is refilled by the next iteration's copy
          continue;
        }
      }
      __syncthreads();  // k has been read: its buffer takes this tile's dk for full-row accesses
#pragma unroll
      for (int nt = 0; nt < D / 8; ++nt) {
        const int col = nt * 8 + 2 * tq;
        *reinterpret_cast<uint32_t*>(&kt.e[warp * 16 + gq][col]) = pack_bf16(dk[nt][0] * s.scale, dk[nt][1] * s.scale);
        *reinterpret_cast<uint32_t*>(&kt.e[warp * 16 + gq + 8][col]) = pack_bf16(dk[nt][2] * s.scale, dk[nt][3] * s.scale);
      }
      __syncthreads();
      for (int i = tid; i < kKeys * (D / 8); i += kThreads) {
        const int row = i / (D / 8), c = i % (D / 8);
        if (s0 + row >= s.S) continue;
        __nv_bfloat16* p = dkb + (int64_t)(s0 + row) * a.dk.ss + c * 8;
        uint4 x = *reinterpret_cast<const uint4*>(&kt.e[row][c * 8]);
        if (add) {
          float v[8], o[8];
          load8(&kt.e[row][c * 8], v);
          load8(&old.e[row][c * 8], o);
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] += o[j];
          store8(p, v);
        } else {
          *reinterpret_cast<uint4*>(p) = x;
        }
      }
      __syncthreads();
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int rr = warp * 16 + gq + 8 * h;
      if (rr >= nrow) continue;
      float* d = a.dq32 + ((int64_t)(b * s.N + g * G) * s.R + r0 + rr) * D + 2 * tq;
#pragma unroll
      for (int nt = 0; nt < D / 8; ++nt) atomicAdd(reinterpret_cast<float2*>(d + nt * 8), make_float2(dq[nt][2 * h], dq[nt][2 * h + 1]));
    }
  }
}

// fp32: the same walk on CUDA cores.  Thread (ty, tx) owns slots (dk) and pairs (dq) ty + 16 i and D / 16 elements.
template <int D>
__global__ void __launch_bounds__(kThreadsF) raw_bwd_f32_kernel(RawBwdArgs a) {
  constexpr int E = D / 16;  // elements of head_dim per thread: tx * 4 + {0..3} (+ 64)
  extern __shared__ __align__(16) float fsm[];
  float* qt = fsm;               // [64][D]
  float* kt = qt + 64 * D;       // [64][D]
  float* gt = kt + 64 * D;       // [64 pairs][65]
  const ScoreArgs& s = a.s;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const int G = s.N / s.Nk, GR = G * s.R;
  const int b = blockIdx.y / s.Nk, g = blockIdx.y % s.Nk;
  const int n_tiles = (s.S + kKeys - 1) / kKeys;
  const float* kb = reinterpret_cast<const float*>(s.k.ptr) + (int64_t)b * s.k.sb + (int64_t)g * s.k.sh;
  float* dkb = reinterpret_cast<float*>(a.dk.ptr) + (int64_t)b * a.dk.sb + (int64_t)g * a.dk.sh;
  const float* gb = reinterpret_cast<const float*>(a.d_raw) + (int64_t)(b * s.N + g * G) * s.R * s.S;
  for (int r0 = 0; r0 < GR; r0 += 64) {
    const int nrow = min(64, GR - r0);
    __syncthreads();
    for (int i = tid; i < 64 * (D / 4); i += kThreadsF) {
      const int rr = i / (D / 4), d = i % (D / 4) * 4, row = min(r0 + rr, GR - 1);
      const float4 x = load4(reinterpret_cast<const float*>(s.q.ptr) + (int64_t)b * s.q.sb + (int64_t)(g * G + row / s.R) * s.q.sh +
                             (int64_t)(s.S - s.R + row % s.R) * s.q.ss + d);
      // (zeros behind the last pair and the last slot: their weights are zero, but an infinity would make NaN of it)
      *reinterpret_cast<float4*>(qt + rr * D + d) = rr < nrow ? x : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float dq[4][E] = {};
    for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
      const int s0 = tile * kKeys;
      __syncthreads();
      for (int i = tid; i < kKeys * (D / 4); i += kThreadsF) {
        const int row = i / (D / 4), d = i % (D / 4) * 4;
        const float4 x = load4(kb + (int64_t)min(s0 + row, s.S - 1) * s.k.ss + d);
        *reinterpret_cast<float4*>(kt + row * D + d) = s0 + row < s.S ? x : make_float4(0.f, 0.f, 0.f, 0.f);
      }
      for (int i = tid; i < 64 * kKeys; i += kThreadsF) {
        const int rr = i / kKeys, c = i % kKeys;
        gt[rr * 65 + c] = rr < nrow && s0 + c < s.S ? gb[(int64_t)(r0 + rr) * s.S + s0 + c] : 0.f;
      }
      __syncthreads();
      float dk[4][E] = {};
      for (int j = 0; j < 64; ++j) {  // j: a pair for dk, a slot for dq
        float qx[E], kx[E];
#pragma unroll
        for (int e = 0; e < E; e += 4) {
          *reinterpret_cast<float4*>(&qx[e]) = *reinterpret_cast<const float4*>(qt + j * D + tx * 4 + e * 16);
          *reinterpret_cast<float4*>(&kx[e]) = *reinterpret_cast<const float4*>(kt + j * D + tx * 4 + e * 16);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float gs = gt[j * 65 + ty + 16 * i], gp = gt[(ty + 16 * i) * 65 + j];
#pragma unroll
          for (int e = 0; e < E; ++e) {
            dk[i][e] = fmaf(gs, qx[e], dk[i][e]);
            dq[i][e] = fmaf(gp, kx[e], dq[i][e]);
          }
        }
      }
      const bool add = a.add || r0 > 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int sl = s0 + ty + 16 * i;
        if (sl >= s.S) continue;
#pragma unroll
        for (int e = 0; e < E; e += 4) {
          float* p = dkb + (int64_t)sl * a.dk.ss + tx * 4 + e * 16;
          float4 v = make_float4(dk[i][e] * s.scale, dk[i][e + 1] * s.scale, dk[i][e + 2] * s.scale, dk[i][e + 3] * s.scale);
          if (add) {
            const float4 o = load4(p);
            v = make_float4(v.x + o.x, v.y + o.y, v.z + o.z, v.w + o.w);
          }
          store4(p, v);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (ty + 16 * i >= nrow) continue;
      float* d = a.dq32 + ((int64_t)(b * s.N + g * G) * s.R + r0 + ty + 16 * i) * D + tx * 4;
#pragma unroll
      for (int e = 0; e < E; ++e) atomicAdd(d + (e & ~3) * 16 + (e & 3), dq[i][e]);
    }
  }
}

// dq32 -> the last R rows of dq: one thread per four elements
template <typename T>
__global__ void __launch_bounds__(256) raw_bwd_rows_kernel(RawBwdArgs a, int D) {
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x, n4 = (int64_t)a.s.B * a.s.N * a.s.R * (D / 4);
  if (i >= n4) return;
  const int d = (int)(i % (D / 4)) * 4;
  const int64_t row = i / (D / 4);
  const int r = (int)(row % a.s.R), n = (int)(row / a.s.R % a.s.N), b = (int)(row / ((int64_t)a.s.R * a.s.N));
  float4 v = load4(a.dq32 + row * D + d);
  v = make_float4(v.x * a.s.scale, v.y * a.s.scale, v.z * a.s.scale, v.w * a.s.scale);
  T* p = reinterpret_cast<T*>(a.dq.ptr) + (int64_t)b * a.dq.sb + (int64_t)n * a.dq.sh + (int64_t)(a.s.S - a.s.R + r) * a.dq.ss + d;
  if (a.add) {
    const float4 o = load4(p);
    v = make_float4(v.x + o.x, v.y + o.y, v.z + o.z, v.w + o.w);
  }
  store4(p, v);
}

// CTAs per (prompt, KV head) so that the grid is resident at once at `per_sm` CTAs per SM
int tiles_grid(int S, int bg, int per_sm) {
  const int n_tiles = (S + kKeys - 1) / kKeys;
  return std::max(1, std::min(n_tiles, per_sm * std::max(1, sm_count()) / bg));
}

}  // namespace

int raw_scores_launch(const brk_score_params& p, void* out, cudaStream_t st) {
  int rc = check_score_params(p);
  if (rc) return rc;
  BRK_REQUIRE(out != nullptr, BRK_E_ARG, "out is null");
  BRK_REQUIRE(p.R <= p.S, BRK_E_ARG, "R=%d exceeds S=%d", p.R, p.S);
  const ScoreArgs a = make_score_args(p);
  // 0.7 * lowest finite value of the dtype, computed the way the reference does (python float -> dtype)
  if (p.dtype == BRK_BF16) {
    const float neg = 0.7f * -3.3895313892515355e38f;
    const dim3 grid(tiles_grid(p.S, p.B * p.Nk, p.D == 128 ? kRawPerSm<128> : kRawPerSm<64>), p.B * p.Nk);
    const size_t sm = p.M <= kMaxSharedSpans ? (size_t)p.M * 8 : 0;
    const int wide = ((uintptr_t)out & 15) == 0 && p.S % 8 == 0;  // eight logits per store; `out` may have any alignment
    return p.D == 128 ? launch_dependent(raw_scores_mma_kernel<128>, grid, dim3(kThreads), sm, st, a, (__nv_bfloat16*)out, neg, wide)
                      : launch_dependent(raw_scores_mma_kernel<64>, grid, dim3(kThreads), sm, st, a, (__nv_bfloat16*)out, neg, wide);
  } else {
    const float neg = (float)(0.7 * -3.4028234663852886e38);
    const dim3 grid((p.S + kKeys - 1) / kKeys, p.B * p.Nk);
    const int sm = 2 * 64 * (p.D + 4) * (int)sizeof(float);
    if (p.D == 128) {
      BRK_CUDA(cudaFuncSetAttribute(raw_scores_f32_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm));
      raw_scores_f32_kernel<128><<<grid, kThreadsF, sm, st>>>(a, (float*)out, neg);
    } else {
      raw_scores_f32_kernel<64><<<grid, kThreadsF, sm, st>>>(a, (float*)out, neg);
    }
  }
  BRK_LAUNCHED();
  return BRK_OK;
}

static size_t raw_dq_bytes(const brk_score_params& p) { return (size_t)p.B * p.N * p.R * p.D * sizeof(float); }
size_t raw_scores_bwd_workspace(const brk_score_params& p) {
  const bool passes = p.dtype == BRK_BF16 && p.Nk > 0 && (p.N / p.Nk) * p.R > kRowsPass;
  const size_t tiles = (size_t)p.B * p.Nk * ((p.S + kKeys - 1) / kKeys);
  return raw_dq_bytes(p) + (passes ? tiles * kKeys * p.D * sizeof(float) : 0);
}

int raw_scores_bwd_launch(const brk_score_params& p, const void* d_raw, const brk_view& dq, const brk_view& dk,
                          int accumulate, void* ws, size_t ws_bytes, cudaStream_t st) {
  int rc = check_score_params(p);
  if (rc) return rc;
  const int al = p.dtype == BRK_BF16 ? 8 : 4;
  BRK_REQUIRE(d_raw && dq.ptr && dk.ptr, BRK_E_ARG, "d_raw / dq / dk is null");
  BRK_REQUIRE(p.R <= p.S, BRK_E_ARG, "R=%d exceeds S=%d", p.R, p.S);
  BRK_REQUIRE((((uintptr_t)d_raw | (uintptr_t)dq.ptr | (uintptr_t)dk.ptr) & 15) == 0 && dq.stride_s % al == 0 &&
                  dq.stride_h % al == 0 && dq.stride_b % al == 0 && dk.stride_s % al == 0 && dk.stride_h % al == 0 &&
                  dk.stride_b % al == 0,
              BRK_E_ARG, "d_raw and the rows of dq / dk must be 16-byte aligned");
  BRK_REQUIRE(ws != nullptr && ws_bytes >= raw_scores_bwd_workspace(p) && ((uintptr_t)ws & 15) == 0, BRK_E_WORKSPACE,
              "workspace %zu < %zu bytes (or not 16-byte aligned)", ws_bytes, raw_scores_bwd_workspace(p));
  RawBwdArgs a;
  a.s = make_score_args(p);
  a.dq = make_view(dq);
  a.dk = make_view(dk);
  a.d_raw = d_raw;
  a.dq32 = reinterpret_cast<float*>(ws);
  a.add = accumulate;
  a.dk32 = reinterpret_cast<float2*>(static_cast<unsigned char*>(ws) + raw_dq_bytes(p));
  BRK_CUDA(cudaMemsetAsync(ws, 0, raw_dq_bytes(p), st));
  const int64_t n4 = (int64_t)p.B * p.N * p.R * (p.D / 4);
  const unsigned rows_grid = (unsigned)((n4 + 255) / 256);
  if (p.dtype == BRK_BF16) {
    const dim3 grid(tiles_grid(p.S, p.B * p.Nk, 2), p.B * p.Nk);
    auto go = [&](auto kern, size_t sm) -> int {
      BRK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
      kern<<<grid, kThreads, sm, st>>>(a);
      BRK_LAUNCHED();
      return BRK_OK;
    };
    rc = p.D == 128 ? go(raw_bwd_mma_kernel<128>, sizeof(MmaTile<128>) + 2 * sizeof(RawBwdStage<128>))
                    : go(raw_bwd_mma_kernel<64>, sizeof(MmaTile<64>) + 2 * sizeof(RawBwdStage<64>));
    if (rc) return rc;
    raw_bwd_rows_kernel<__nv_bfloat16><<<rows_grid, 256, 0, st>>>(a, p.D);
  } else {
    const dim3 grid(tiles_grid(p.S, p.B * p.Nk, 2), p.B * p.Nk);
    const int sm = (2 * 64 * p.D + 64 * 65) * (int)sizeof(float);
    auto go = [&](auto kern) -> int {
      BRK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, sm));
      kern<<<grid, kThreadsF, sm, st>>>(a);
      BRK_LAUNCHED();
      return BRK_OK;
    };
    rc = p.D == 128 ? go(raw_bwd_f32_kernel<128>) : go(raw_bwd_f32_kernel<64>);
    if (rc) return rc;
    raw_bwd_rows_kernel<float><<<rows_grid, 256, 0, st>>>(a, p.D);
  }
  BRK_LAUNCHED();
  return BRK_OK;
}

}  // namespace brk
