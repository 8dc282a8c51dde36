// Score extraction for BlockRank ranking: HBM-bound skinny products of a few
// signal rows of Q against every document key.
//
//   doc_partial_kernel   one CTA per (document, prompt, KV head): each thread
//                        owns whole key rows (read once per KV head, shared by
//                        the G query heads of the group) and keeps an online
//                        (max, sum-exp) per signal row; the CTA writes one
//                        (max, sum) pair per (head, row, document).  fp32 inputs.
//   doc_partial_mma_kernel  the same for bf16, a CTA walking through several documents
//                        of one (prompt, KV head): the (G*R signal rows) x (keys)
//                        products go through warp-level mma (m16n8k16), key
//                        rows straight from global memory into the B fragments,
//                        requested one group ahead across document boundaries.
//                        The product is 8-16 rows tall and bound by the K read;
//                        a tcgen05 tile (M >= 64, operands staged in shared
//                        memory, result through tensor memory) would add
//                        latency to a kernel that has no tensor-rate problem.
//   doc_merge_kernel     one CTA per prompt, or a cluster of up to eight for many pairs, brought up as the partial kernel's
//                        CTAs leave the SMs: merges the per-document pairs into the softmax over all document tokens, emits
//                        the per-document probability mass and then the mean over heads and rows / temperature.  As the job
//                        of the last CTA of a prompt, found by counters that a memset cleared in front, with a fence and an
//                        atomic in every CTA: 4 prompts of 100 documents 37.4 us, now 29.1 (the K read at 5.4 TB/s), one
//                        prompt of 100 20.5, now 13.7.  A call of a few short documents: alone 20.5, now 19.2; in a row,
//                        bound by the host, 12.3 and 9.2.
#include <algorithm>
#include <atomic>

#include "brk_common.cuh"
#include "mma_bf16.cuh"
#include "score_args.cuh"
#include "tc_ptx.cuh"

namespace brk {
namespace {

constexpr int kThreads = 160;  // five warps: a 160-token document is one pass
constexpr int kRowBatch = 8;  // signal rows accumulated per pass over a key
constexpr int kKeyStages = 4;   // asynchronous key-row copies a lane keeps in flight in the bf16 kernel
constexpr int kDocsPerCta = 64;  // documents one CTA of the bf16 kernel walks through, at most


__device__ __forceinline__ void merge_ml(float& m, float& l, float m2, float l2) {
  const float mn = fmaxf(m, m2);
  const float ref = (mn == -INFINITY) ? 0.f : mn;
  l = l * exp2f(m - ref) + l2 * exp2f(m2 - ref);
  m = mn;
}

// two more logits (already in log2 units; -inf = masked) into a running (max, sum)
__device__ __forceinline__ void merge_pair(float& m, float& l, float x0, float x1) {
  const float mn = fmaxf(m, fmaxf(x0, x1));
  const float ref = (mn == -INFINITY) ? 0.f : mn;
  l = l * exp2f(m - ref) + (exp2f(x0 - ref) + exp2f(x1 - ref));
  m = mn;
}

// One CTA per prompt, or a cluster of them (kCluster: grid.x) that share its KV heads.  A warp takes two (head, signal row)
// pairs at a time, so that their statistics travel together; then the masses are summed per document, group by group of heads,
// in a fixed order, the same for any number of CTAs.  Bound by latency: a read of the pairs, a write and a read of the masses.
// (Clusters of 512 threads at 64 registers, so that two CTAs share an SM: at 78 registers 32 prompts of 300 documents took 196
// us, now 185; one row at a time, no spill, 2,000 documents with 16 rows 277, now 248.)
template <bool kCluster>
constexpr int merge_threads = kCluster ? 512 : 1024;
template <bool kCluster>
__global__ void __launch_bounds__(merge_threads<kCluster>, kCluster ? 2 : 1) doc_merge_kernel(ScoreArgs a) {
  constexpr int kMergeThreads = merge_threads<kCluster>;
  constexpr int kHeld = 8;  // pairs per lane kept in registers: one round trip per row up to 256 documents
  constexpr int kWarps = kMergeThreads / 32, kRows = 2;
  __shared__ float s_group[kMergeThreads];
  ptx::grid_dependency_wait();  // the partial kernel's pairs
  const int nd = a.M - 2, b = kCluster ? blockIdx.y : blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // KV heads of this CTA: g_lo .. g_lo + n_g - 1, of `per` in all but the last ones (a.Nk spelled out below where there is one
  // CTA: kept in a variable from here on, it made the kernel spill)
  const int n_cta = kCluster ? (int)gridDim.x : 1, rank = kCluster ? (int)blockIdx.x : 0;
  const int per = kCluster ? (a.Nk + n_cta - 1) / n_cta : 0;
  const int g_lo = min(a.Nk, rank * per), n_g = kCluster ? min(a.Nk, g_lo + per) - g_lo : 0;
  const int G = a.N / a.Nk, GR = G * a.R, W = kCluster ? n_g * GR : a.N * a.R;
  const size_t w0 = kCluster ? ((size_t)b * a.Nk + g_lo) * GR : (size_t)b * W;
  for (int first = warp; first < W; first += kRows * kWarps) {
    float2 held[kRows][kHeld];
    float mx[kRows], z[kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const float2* const p = a.partial + (w0 + first + r * kWarps) * nd;
      const bool on = first + r * kWarps < W;
#pragma unroll
      for (int i = 0; i < kHeld; ++i) held[r][i] = on && lane + 32 * i < nd ? p[lane + 32 * i] : make_float2(-INFINITY, 0.f);
    }
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const float2* const p = a.partial + (w0 + first + r * kWarps) * nd;
      const int n = first + r * kWarps < W ? nd : 0;
      mx[r] = -INFINITY;
#pragma unroll
      for (int i = 0; i < kHeld; ++i) mx[r] = fmaxf(mx[r], held[r][i].x);
      for (int d = lane + 32 * kHeld; d < n; d += 32) mx[r] = fmaxf(mx[r], p[d].x);
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], off));
      const float ref = (mx[r] == -INFINITY) ? 0.f : mx[r];
      z[r] = 0.f;
#pragma unroll
      for (int i = 0; i < kHeld; ++i) {
        held[r][i].y *= exp2f(held[r][i].x - ref);  // un-normalised mass of the document
        z[r] += held[r][i].y;
      }
      for (int d = lane + 32 * kHeld; d < n; d += 32) z[r] += p[d].y * exp2f(p[d].x - ref);
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) z[r] += __shfl_xor_sync(0xffffffffu, z[r], off);
      const float inv = z[r] > 0.f ? 1.f / z[r] : 0.f;
      float* const mass = a.mass + (w0 + first + r * kWarps) * nd;
#pragma unroll
      for (int i = 0; i < kHeld; ++i)
        if (lane + 32 * i < n) mass[lane + 32 * i] = held[r][i].y * inv;
      for (int d = lane + 32 * kHeld; d < n; d += 32) mass[d] = p[d].y * exp2f(p[d].x - ref) * inv;
    }
  }
  if (a.logits == nullptr) return;
  __syncthreads();  // every mass of these heads has been written
  // A thread sums a group's rows for one document, then one thread per document the groups of all CTAs, in order.
  const int tile = max(1, kMergeThreads / (kCluster ? per : a.Nk));  // documents at a time
  for (int d0 = 0; d0 < nd; d0 += tile) {
    const int n = min(tile, nd - d0);
    float total = 0.f;
    for (int g0 = 0; g0 < (kCluster ? per : a.Nk); g0 += kMergeThreads) {  // (more groups than threads: in rounds)
      const int ng = min((kCluster ? per : a.Nk) - g0, kMergeThreads);
      const int g = tid / n, d = tid % n;
      if (g < (kCluster ? min(ng, n_g - g0) : ng)) {
        const float* const m = a.mass + (w0 + (size_t)(g0 + g) * GR) * nd + d0 + d;
        float acc = 0.f;
#pragma unroll 8
        for (int row = 0; row < GR; ++row) acc += m[(size_t)row * nd];
        s_group[g * n + d] = acc;
      }
      if (kCluster) ptx::cluster_sync(); else __syncthreads();
      if (kCluster) {
        if (tid < n && tid % n_cta == rank)
          for (int c = 0; c < n_cta; ++c) {
            const int left = min(ng, a.Nk - c * per - g0);  // of CTA c's groups in this round
            for (int i = 0; i < left; ++i) total += ptx::ld_cluster_f32(ptx::smem_u32(s_group + i * n + tid), c);
          }
      } else if (tid < n) {
        for (int i = 0; i < ng; ++i) total += s_group[i * n + tid];
      }
      if (kCluster) ptx::cluster_sync(); else __syncthreads();
    }
    if (tid < n && (!kCluster || tid % n_cta == rank)) a.logits[(size_t)b * nd + d0 + tid] = total * a.inv_count_temp;
  }
}

// dot products of one key row against kRowBatch staged query rows
template <typename T, int D>
__device__ __forceinline__ void key_dots(const T* __restrict__ kp, const float* __restrict__ qs, int nrows,
                                         float (&acc)[kRowBatch]) {
#pragma unroll
  for (int i = 0; i < kRowBatch; ++i) acc[i] = 0.f;
#pragma unroll 4
  for (int d = 0; d < D; d += 4) {
    const float4 kv = load4(kp + d);
#pragma unroll
    for (int i = 0; i < kRowBatch; ++i) {
      if (i < nrows) {
        const float4 qv = *reinterpret_cast<const float4*>(qs + i * D + d);
        acc[i] = fmaf(qv.x, kv.x, acc[i]);
        acc[i] = fmaf(qv.y, kv.y, acc[i]);
        acc[i] = fmaf(qv.z, kv.z, acc[i]);
        acc[i] = fmaf(qv.w, kv.w, acc[i]);
      }
    }
  }
}

// One CTA per (document, prompt, KV head).  Each warp stages 32 key rows at a time in shared memory
// with fully coalesced 16-byte loads (all in flight together), then every lane owns one key: its
// dot products against the G*R staged query rows read the key from shared memory (row stride padded
// by 16 bytes, conflict-free for 16-byte accesses) and the query rows as broadcasts.  (head_dim 64 spills 16 bytes at the 96
// registers that it is given; with 128 and next to no spill, but fewer CTAs per SM, 4 prompts of 100 documents take 81 us, not 62.)
template <typename T, int D>
__global__ void __launch_bounds__(kThreads) doc_partial_kernel(ScoreArgs a) {
  constexpr int kRowBytes = D * (int)sizeof(T);
  constexpr int kPitch = kRowBytes + 16;
  constexpr int kChunks = kRowBytes / 16;  // 16-byte pieces per key row
  ptx::grid_dependency_wait();    // (a call's launch overlaps the end of what is in front of it, the merge of the call before for one)
  ptx::grid_dependency_launch();  // the merge kernel may be brought up once every CTA is at work
  extern __shared__ __align__(16) float smem[];
  const int G = a.N / a.Nk;
  const int GR = G * a.R;
  float* qs = smem;                                    // [GR][D], scaled by scale*log2(e)
  float2* red = reinterpret_cast<float2*>(qs + GR * D);  // [kThreads/32][kRowBatch]
  unsigned char* ktile = reinterpret_cast<unsigned char*>(red + (kThreads / 32) * kRowBatch);  // [warps][32][kPitch]

  const int nd = a.M - 2;
  const int d = blockIdx.x;
  const int b = blockIdx.y / a.Nk, g = blockIdx.y % a.Nk;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int start = a.blk_start[(size_t)b * a.M + 1 + d];
  const int len = a.blk_len[(size_t)b * a.M + 1 + d];

  const float sl2 = a.scale * 1.4426950408889634f;
  for (int i = tid; i < GR * (D / 4); i += kThreads) {
    const int row = i / (D / 4), d4 = i % (D / 4);
    const int hl = row / a.R, r = row % a.R;
    const int slot = a.rows[b * a.R + r];
    const T* qp = reinterpret_cast<const T*>(a.q.ptr) + (int64_t)b * a.q.sb + (int64_t)(g * G + hl) * a.q.sh +
                  (int64_t)slot * a.q.ss;
    float4 x = load4(qp + d4 * 4);
    *reinterpret_cast<float4*>(qs + row * D + d4 * 4) = make_float4(x.x * sl2, x.y * sl2, x.z * sl2, x.w * sl2);
  }
  __syncthreads();

  const unsigned char* kb = reinterpret_cast<const unsigned char*>(
      reinterpret_cast<const T*>(a.k.ptr) + (int64_t)b * a.k.sb + (int64_t)g * a.k.sh);
  const int64_t row_stride = a.k.ss * (int64_t)sizeof(T);
  unsigned char* my_tile = ktile + (size_t)warp * 32 * kPitch;
  for (int r0 = 0; r0 < GR; r0 += kRowBatch) {
    const int nrows = min(kRowBatch, GR - r0);
    float m[kRowBatch], l[kRowBatch];
#pragma unroll
    for (int i = 0; i < kRowBatch; ++i) { m[i] = -INFINITY; l[i] = 0.f; }
    for (int base = warp * 32; base < len; base += kThreads) {
      const int nkeys = min(32, len - base);
      __syncwarp();
#pragma unroll
      for (int i = 0; i < kChunks; ++i) {
        const int idx = lane + 32 * i, row = idx / kChunks, ch = idx % kChunks;
        if (row < nkeys)
          *reinterpret_cast<uint4*>(my_tile + row * kPitch + ch * 16) =
              *reinterpret_cast<const uint4*>(kb + (int64_t)(start + base + row) * row_stride + ch * 16);
      }
      __syncwarp();
      if (lane < nkeys) {
        float acc[kRowBatch];
        key_dots<T, D>(reinterpret_cast<const T*>(my_tile + lane * kPitch), qs + r0 * D, nrows, acc);
#pragma unroll
        for (int i = 0; i < kRowBatch; ++i)
          if (i < nrows) merge_ml(m[i], l[i], acc[i], 1.f);
      }
    }
    // warp then CTA reduction, fixed order
#pragma unroll
    for (int i = 0; i < kRowBatch; ++i) {
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        const float m2 = __shfl_xor_sync(0xffffffffu, m[i], off);
        const float l2 = __shfl_xor_sync(0xffffffffu, l[i], off);
        merge_ml(m[i], l[i], m2, l2);
      }
    }
    __syncthreads();
    if (lane == 0) {
#pragma unroll
      for (int i = 0; i < kRowBatch; ++i) red[warp * kRowBatch + i] = make_float2(m[i], l[i]);
    }
    __syncthreads();
    if (tid < nrows) {
      float mm = -INFINITY, ll = 0.f;
      for (int w = 0; w < kThreads / 32; ++w) {
        const float2 x = red[w * kRowBatch + tid];
        merge_ml(mm, ll, x.x, x.y);
      }
      const int row = r0 + tid;
      const int n = g * G + row / a.R, r = row % a.R;
      a.partial[(((size_t)b * a.N + n) * a.R + r) * nd + d] = make_float2(mm, ll);
    }
  }
}

// bf16 version of doc_partial_kernel on warp-level MMA.  One CTA per (document, prompt, KV head);
// a warp takes 8 keys at a time: C[16 signal rows x 8 keys] += Q[16 x 16] K^T[16 x 8] over D/16
// steps.  Lane (q = lane/4, j = lane%4) reads 16 bytes (8 elements of d) of key q per 32 elements
// of d, which is exactly its B fragment for two consecutive k-steps when the contraction index is
// taken in the order (8j+0,1 | 8j+2,3) then (8j+4,5 | 8j+6,7); the A fragments (signal rows q and
// q+8) are read from Q with the same 16-byte pattern, so both operands come straight from global
// memory with fully used sectors and no shared-memory staging.
template <int D>
__global__ void __launch_bounds__(kThreads, 4) doc_partial_mma_kernel(ScoreArgs a) {
  constexpr int kSteps = D / 32;
  constexpr int kStride = (kThreads / 32) * 8;
  __shared__ float2 red[2][kThreads / 32][16];
  __shared__ int s_start[kDocsPerCta], s_len[kDocsPerCta];
  __shared__ uint4 ring[kKeyStages][kSteps][kThreads];  // every lane copies into and reads back its own 16-byte cells
  ptx::grid_dependency_wait();    // (a call's launch overlaps the end of what is in front of it, the merge of the call before for one)
  ptx::grid_dependency_launch();  // the merge kernel may be brought up once every CTA is at work
  const int G = a.N / a.Nk;
  const int GR = G * a.R;
  const int nd = a.M - 2;
  const int b = blockIdx.y / a.Nk, g = blockIdx.y % a.Nk;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int qr = lane >> 2, j = lane & 3;
  const float sl2 = a.scale * 1.4426950408889634f;
  const __nv_bfloat16* kbase = reinterpret_cast<const __nv_bfloat16*>(a.k.ptr) + (int64_t)b * a.k.sb + (int64_t)g * a.k.sh;

  // This CTA's documents: blockIdx.x, blockIdx.x + gridDim.x, ... (the launch keeps them within kDocsPerCta).
  const int n_mine = (nd - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  for (int i = tid; i < n_mine; i += kThreads) {
    const int d = blockIdx.x + i * gridDim.x;
    s_start[i] = a.blk_start[(size_t)b * a.M + 1 + d];
    s_len[i] = a.blk_len[(size_t)b * a.M + 1 + d];
  }
  __syncthreads();

  unsigned red_par = 0;
  for (int r0 = 0; r0 < GR; r0 += 16) {
    // A warp visits the 8-key groups (document i, keys base..base+7), base = 8*warp, 8*warp + 40, ..., of
    // every document of the CTA in order.  The key rows travel through a ring of kKeyStages asynchronous
    // copies per lane (16 bytes each, global -> shared, read back by the lane that requested them), issued
    // kKeyStages - 1 groups ahead of the products and across document boundaries: the kernel is bound by the
    // latency of these loads, and this is what keeps enough of them in flight.
    const bool has_hi = r0 + 8 < GR;  // with 8 or fewer (head, signal row) pairs left, rows 8..15 of the product are padding
    int ci = -1, cbase = 0, clen = 0;  // the group requested next: keys cbase.. of the CTA's document ci (clen keys)
    const __nv_bfloat16* cptr = kbase;  // first key row of that document, this lane's 16-byte column
    auto request = [&](int stage) {
      while (ci < n_mine && cbase >= clen) {  // next document that still has a group for this warp
        ++ci;
        cbase = warp * 8;
        clen = ci < n_mine ? s_len[ci] : 0;
        if (ci < n_mine) cptr = kbase + (int64_t)s_start[ci] * a.k.ss + 8 * j;
      }
      if (ci < n_mine) {
        const int key = min(cbase + qr, clen - 1);  // rows past the end re-read the last key; their columns are dropped below
        const __nv_bfloat16* kp = cptr + (int64_t)key * a.k.ss;
#pragma unroll
        for (int st = 0; st < kSteps; ++st) cp_async16(&ring[stage][st][tid], kp + 32 * st);
        cbase += kStride;
      }
      cp_async_commit();  // (an empty group when the documents are exhausted: the count below stays uniform)
    };
#pragma unroll
    for (int s = 0; s < kKeyStages - 1; ++s) request(s);
    // (the signal rows of Q are read behind the first key requests: both latencies overlap)
    uint4 qa[kSteps], qb[kSteps];  // signal rows r0+qr and r0+qr+8
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int row = r0 + qr + 8 * h;
      const bool ok = row < GR;
      const int hl = ok ? row / a.R : 0, r = ok ? row % a.R : 0;
      const int slot = a.rows[b * a.R + r];
      const __nv_bfloat16* qp = reinterpret_cast<const __nv_bfloat16*>(a.q.ptr) + (int64_t)b * a.q.sb +
                                (int64_t)(g * G + hl) * a.q.sh + (int64_t)slot * a.q.ss + 8 * j;
#pragma unroll
      for (int st = 0; st < kSteps; ++st) {
        const uint4 v = ok ? *reinterpret_cast<const uint4*>(qp + 32 * st) : make_uint4(0, 0, 0, 0);
        if (h == 0) qa[st] = v; else qb[st] = v;
      }
    }
    int stage_r = 0, stage_w = kKeyStages - 1;
    for (int i = 0; i < n_mine; ++i) {
      const int len = s_len[i];
      float m_lo = -INFINITY, l_lo = 0.f, m_hi = -INFINITY, l_hi = 0.f;
      for (int base = warp * 8; base < len; base += kStride) {
        request(stage_w);
        stage_w = stage_w + 1 == kKeyStages ? 0 : stage_w + 1;
        cp_async_wait<kKeyStages - 1>();  // the oldest group -- this one -- has landed
        uint4 kf[kSteps];
#pragma unroll
        for (int st = 0; st < kSteps; ++st) kf[st] = ring[stage_r][st][tid];
        stage_r = stage_r + 1 == kKeyStages ? 0 : stage_r + 1;
        float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int st = 0; st < kSteps; ++st) {
          mma16816(c, {qa[st].x, qb[st].x, qa[st].y, qb[st].y}, kf[st].x, kf[st].y);
          mma16816(c, {qa[st].z, qb[st].z, qa[st].w, qb[st].w}, kf[st].z, kf[st].w);
        }
        // c[0], c[1]: row qr, keys base + 2j, 2j + 1; c[2], c[3]: row qr + 8, same keys
        const bool ok0 = base + 2 * j < len, ok1 = base + 2 * j + 1 < len;
        merge_pair(m_lo, l_lo, ok0 ? c[0] * sl2 : -INFINITY, ok1 ? c[1] * sl2 : -INFINITY);
        if (has_hi) merge_pair(m_hi, l_hi, ok0 ? c[2] * sl2 : -INFINITY, ok1 ? c[3] * sl2 : -INFINITY);
      }
      // the four lanes of a row, then the warps, in a fixed order
#pragma unroll
      for (int off = 1; off <= 2; off <<= 1) {
        const float m2 = __shfl_xor_sync(0xffffffffu, m_lo, off), l2 = __shfl_xor_sync(0xffffffffu, l_lo, off);
        merge_ml(m_lo, l_lo, m2, l2);
        if (has_hi) {
          const float m3 = __shfl_xor_sync(0xffffffffu, m_hi, off), l3 = __shfl_xor_sync(0xffffffffu, l_hi, off);
          merge_ml(m_hi, l_hi, m3, l3);
        }
      }
      // red[] alternates between documents: a buffer is rewritten two documents later, behind the barrier of
      // the document in between, which its readers reach only after reading it
      float2 (&rd)[kThreads / 32][16] = red[red_par];
      red_par ^= 1u;
      if (j == 0) {
        rd[warp][qr] = make_float2(m_lo, l_lo);
        rd[warp][qr + 8] = make_float2(m_hi, l_hi);
      }
      __syncthreads();
      if (tid < 16 && r0 + tid < GR) {
        float mm = -INFINITY, ll = 0.f;
        for (int w = 0; w < kThreads / 32; ++w) merge_ml(mm, ll, rd[w][tid].x, rd[w][tid].y);
        const int row = r0 + tid;
        const int n = g * G + row / a.R, r = row % a.R;
        const int d = blockIdx.x + i * gridDim.x;
        a.partial[(((size_t)b * a.N + n) * a.R + r) * nd + d] = make_float2(mm, ll);
      }
    }
  }
}

}  // namespace

// scratch: the [B, N, R, nd] (max, sum) pairs
static size_t partial_bytes(const brk_score_params& p) {
  const size_t nd = p.M > 2 ? p.M - 2 : 0;
  return (size_t)p.B * p.N * p.R * nd * sizeof(float2);
}

size_t doc_scores_workspace(const brk_score_params& p) { return partial_bytes(p); }

static int doc_scores_run(const brk_score_params& p, void* ws, size_t ws_bytes, cudaStream_t st) {
  int rc = check_score_params(p);
  if (rc) return rc;
  BRK_REQUIRE(p.M >= 3, BRK_E_ARG, "document scores need at least one document block (M=%d)", p.M);
  BRK_REQUIRE(p.rows && p.doc_mass, BRK_E_ARG, "rows / doc_mass must be given");
  BRK_REQUIRE(ws != nullptr && ws_bytes >= partial_bytes(p) && ((uintptr_t)ws & 7) == 0, BRK_E_WORKSPACE,
              "workspace %zu < %zu bytes (or not 8-byte aligned)", ws_bytes, partial_bytes(p));
  BRK_REQUIRE(p.temperature > 0.f, BRK_E_ARG, "temperature must be positive");
  ScoreArgs a = make_score_args(p);
  a.partial = static_cast<float2*>(ws);
  a.mass = p.doc_mass;
  a.logits = p.logits;
  a.inv_count_temp = 1.f / ((float)(p.N * p.R) * p.temperature);
  const int nd = p.M - 2, G = p.N / p.Nk;
  dim3 grid(nd, p.B * p.Nk);
  const size_t pitch = (size_t)p.D * (p.dtype == BRK_BF16 ? 2 : 4) + 16;
  const size_t sm = (size_t)G * p.R * p.D * 4 + (kThreads / 32) * kRowBatch * sizeof(float2) + (kThreads / 32) * 32 * pitch;
  // The merge of one prompt: up to 16,384 pairs on one SM, more on up to eight.  One prompt of 300 documents (19,200 pairs) 31.1
  // us on one, 28.4 on eight, of 500 with 16 signal rows 220 and 133, of 2,000 with 16 rows 600 and 248; 16 prompts of 250
  // (16,000 pairs each) 101 and 104, 4 of 100 (6,400) 29.3 and 30.0.  (With every prompt on one, more than 100,000 pairs took
  // longer than when the CTA of each KV head that finished last merged its rows: 206 us for 500 with 16 rows, 411 for 2,000.)
  int merge_ctas = 1;
  if ((int64_t)p.N * p.R * nd > 16384)
    while (2 * merge_ctas <= std::min(p.Nk, 8)) merge_ctas *= 2;
  auto merge = [&]() -> int {
    if (merge_ctas == 1) return launch_dependent(doc_merge_kernel<false>, dim3(p.B), dim3(merge_threads<false>), 0, st, a);
    return launch_dependent_clusters(merge_ctas, doc_merge_kernel<true>, dim3(merge_ctas, p.B), dim3(merge_threads<true>), 0, st, a);
  };
  auto launch = [&](auto kern) -> int {
    // (the kernels also hold a few KB of static shared memory, which counts against the same 48 KB default)
    if (sm + 8192 > 48 * 1024) BRK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    if ((rc = launch_dependent(kern, grid, dim3(kThreads), sm, st, a))) return rc;
    return merge();
  };
  if (p.dtype == BRK_BF16) {
    // A CTA walks through several documents so that its key loads overlap across document boundaries; the
    // grid is sized to be resident at once (four CTAs per SM) when there are enough documents for that.
    const int slots = 4 * std::max(1, sm_count());
    int per_bg = std::max(1, slots / (p.B * p.Nk));
    per_bg = std::min(nd, std::max(per_bg, (nd + kDocsPerCta - 1) / kDocsPerCta));
    dim3 grid_docs(per_bg, p.B * p.Nk);
    auto run = [&](auto kern, std::atomic<bool>* configured) -> int {
      // Four CTAs with their key rings need 170 KB of shared memory per SM: ask for the large carve-out, once per device.
      int dev = 0;
      BRK_CUDA(cudaGetDevice(&dev));
      if (dev < 0 || dev >= 64 || !configured[dev].load(std::memory_order_acquire)) {
        BRK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared));
        if (dev >= 0 && dev < 64) configured[dev].store(true, std::memory_order_release);
      }
      return launch_dependent(kern, grid_docs, dim3(kThreads), 0, st, a);
    };
    static std::atomic<bool> done128[64] = {}, done64[64] = {};
    rc = p.D == 128 ? run(doc_partial_mma_kernel<128>, done128) : run(doc_partial_mma_kernel<64>, done64);
    if (rc) return rc;
    return merge();
  }
  return p.D == 128 ? launch(doc_partial_kernel<float, 128>) : launch(doc_partial_kernel<float, 64>);
}

int doc_scores_launch(const brk_score_params& p, void* ws, size_t ws_bytes, cudaStream_t st) {
  return doc_scores_run(p, ws, ws_bytes, st);
}

// ---- allocation-free variant ----------------------------------------------------------------
// Scratch for brk_doc_scores_static: the (max, sum) pairs live in this fixed
// array instead of a caller-provided workspace.  It is part of the library image, so every device that
// loads the library holds these bytes until the process exits.
static __device__ __align__(256) unsigned char g_static_scratch[BRK_STATIC_SCRATCH_BYTES];
// The call's limits are those that it had when the array began with 4096 counters: nothing uses these bytes, and what was refused
// stays refused.
constexpr size_t kStaticReserve = 16384;

int doc_scores_static_launch(const brk_score_params& p, cudaStream_t st) {
  int rc = check_score_params(p);  // argument errors are reported as such, before the size test
  if (rc) return rc;
  BRK_REQUIRE(p.M >= 3, BRK_E_ARG, "document scores need at least one document block (M=%d)", p.M);
  BRK_REQUIRE((int64_t)p.B * (p.Nk + 1) <= 4096, BRK_E_WORKSPACE, "brk_doc_scores_static: B*(Nk+1) = %d, at most 4096", p.B * (p.Nk + 1));
  const size_t need = kStaticReserve + partial_bytes(p);
  BRK_REQUIRE(need <= (size_t)BRK_STATIC_SCRATCH_BYTES, BRK_E_WORKSPACE,
              "brk_doc_scores_static: 16384 + B*N*R*(M-2)*8 = %zu bytes of scratch needed, the built-in array holds %zu; "
              "use brk_doc_scores with a caller workspace for this size",
              need, (size_t)BRK_STATIC_SCRATCH_BYTES);
  // In host code the array's name is only a handle; the kernels need its device address, which
  // differs per device.  It is looked up once per device, with that device current; the cache is
  // atomic so that two host threads making their first calls at the same time both end up with
  // the (identical) address.
  static std::atomic<void*> dev_ptr[64];
  int dev = 0;
  BRK_CUDA(cudaGetDevice(&dev));
  BRK_REQUIRE(dev >= 0 && dev < 64, BRK_E_UNSUPPORTED, "device ordinal %d out of range", dev);
  void* ptr = dev_ptr[dev].load(std::memory_order_acquire);
  if (ptr == nullptr) {
    BRK_CUDA(cudaGetSymbolAddress(&ptr, g_static_scratch));
    BRK_REQUIRE(ptr != nullptr, BRK_E_CUDA, "cudaGetSymbolAddress returned a null scratch address");
    dev_ptr[dev].store(ptr, std::memory_order_release);
  }
  // every (prompt, head, row, document) pair is overwritten before it is read: nothing left by an earlier call has to be cleared
  return doc_scores_run(p, ptr, (size_t)BRK_STATIC_SCRATCH_BYTES, st);
}

}  // namespace brk
