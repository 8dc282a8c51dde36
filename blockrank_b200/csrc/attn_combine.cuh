// Merge of the query block's key chunks, shared by the tcgen05 and the fp32 attention kernels.
#pragma once
#include <algorithm>

#include "brk_common.cuh"
#include "tc_ptx.cuh"

namespace brk {

struct CombineArgs {
  View o;
  float* lse;
  const int32_t* blk_start;
  const int32_t* blk_len;
  const int* hdr;
  int B, N, S, M;
  int lq_max, n_split;
  const float* part_o;    // [B, N, lq_max, n_split, HD] un-normalised partial outputs
  const float2* part_ml;  // [B, N, lq_max, n_split] (running max in log2 units, sum)
};

// One warp per (prompt, head, query token) -- of the first 64 tokens, then of the next 64: a padded grid's bound on the
// query block's length is its block size, which few query blocks reach.  Lane c holds the statistics of chunk c (at most 32
// chunks).  Bound by latency: a call has a dozen warps per SM, so a row's statistics and its first U accesses of partial
// rows are requested together (a chunk without keys has written no partial row: its bytes are not used).  With the partial
// rows behind their weights, four at a time, 32 chunks of one prompt took 21 us, now 7.
constexpr int kCombineTokens = 64;
template <typename T, int HD, int U>
__global__ void __launch_bounds__(128) attn_combine_kernel(CombineArgs a) {
  constexpr int kSplit = 128 / HD;  // chunks per warp-wide access
  const int lane = threadIdx.x & 31;
  const int64_t w = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  const int step = min(a.lq_max, kCombineTokens);
  const int n = (int)((w / step) % a.N);
  const int b = (int)(w / ((int64_t)step * a.N));
  ptx::grid_dependency_wait();
  if (b >= a.B) return;
  const int sub = lane / (HD / 4), col = (lane % (HD / 4)) * 4;
  const int bad = a.hdr[1];
  const int start = a.blk_start[(size_t)b * a.M + a.M - 1], len = a.blk_len[(size_t)b * a.M + a.M - 1];
  if (bad != 0) return;
  for (int tok = (int)(w % step); tok < len; tok += step) {
    const int64_t row = ((int64_t)b * a.N + n) * a.lq_max + tok;
    const float* const part = a.part_o + row * a.n_split * HD + col;
    const float2 ml = lane < a.n_split ? a.part_ml[row * a.n_split + lane] : make_float2(-INFINITY, 0.f);
    float4 o[U];
    auto fetch = [&](int c0) {
#pragma unroll
      for (int i = 0; i < U; ++i) {
        const int c = c0 + i * kSplit + sub;
        if (c < a.n_split) o[i] = load4(part + (int64_t)c * HD);
      }
    };
    fetch(0);
    float mx = ml.x;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    const float ref = (mx == -INFINITY) ? 0.f : mx;
    const float wgt = ml.y > 0.f ? exp2f(ml.x - ref) : 0.f;  // chunks that saw no key carry no output
    float l = 0.f;  // (in the order of the chunks, as the rows below: the result does not depend on how the lanes are dealt)
    for (int c = 0; c < a.n_split; ++c)
      l = fmaf(__shfl_sync(0xffffffffu, ml.y, c), __shfl_sync(0xffffffffu, wgt, c), l);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int c0 = 0; c0 < a.n_split; c0 += U * kSplit) {
      if (c0 > 0) fetch(c0);
#pragma unroll
      for (int i = 0; i < U; ++i) {
        const int c = c0 + i * kSplit + sub;
        const float f = __shfl_sync(0xffffffffu, wgt, c & 31);
        if (c < a.n_split && f > 0.f) {
          acc.x = fmaf(o[i].x, f, acc.x); acc.y = fmaf(o[i].y, f, acc.y);
          acc.z = fmaf(o[i].z, f, acc.z); acc.w = fmaf(o[i].w, f, acc.w);
        }
      }
    }
    if (kSplit == 2) {
      acc.x += __shfl_xor_sync(0xffffffffu, acc.x, 16); acc.y += __shfl_xor_sync(0xffffffffu, acc.y, 16);
      acc.z += __shfl_xor_sync(0xffffffffu, acc.z, 16); acc.w += __shfl_xor_sync(0xffffffffu, acc.w, 16);
    }
    const float inv = l > 0.f ? 1.f / l : 0.f;
    T* dst = reinterpret_cast<T*>(a.o.ptr) + (int64_t)b * a.o.sb + (int64_t)(start + tok) * a.o.ss + (int64_t)n * a.o.sh + col;
    if (sub == 0) store4(dst, make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv));
    if (a.lse != nullptr && lane == 0) a.lse[((int64_t)b * a.N + n) * a.S + start + tok] = (ref + log2f(l)) * 0.6931471805599453f;
  }
}

template <typename T, int HD>
int attn_combine_launch(const CombineArgs& c, cudaStream_t st) {
  const int64_t warps = (int64_t)c.B * c.N * std::min(c.lq_max, kCombineTokens);
  const dim3 grid((unsigned)((warps + 3) / 4)), block(128);
  if (c.n_split <= 8) return launch_dependent(attn_combine_kernel<T, HD, 8>, grid, block, 0, st, c);
  return launch_dependent(attn_combine_kernel<T, HD, 16>, grid, block, 0, st, c);
}

}  // namespace brk
