// Merge of the query block's key chunks, shared by the tcgen05 and the fp32 attention kernels.
#pragma once
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

// One warp per (prompt, head, query token); lane c holds the statistics of chunk c (at most 32 chunks).  Bound by latency:
// the partial rows are fetched four chunks at a time (one after another, behind their weights, 26 chunks took 16 us).
template <typename T, int HD>
__global__ void __launch_bounds__(128) attn_combine_kernel(CombineArgs a) {
  constexpr int kSplit = 128 / HD;  // chunks per warp-wide access
  const int lane = threadIdx.x & 31;
  const int64_t w = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  const int tok = (int)(w % a.lq_max);
  const int n = (int)((w / a.lq_max) % a.N);
  const int b = (int)(w / ((int64_t)a.lq_max * a.N));
  ptx::grid_dependency_wait();
  if (b >= a.B || a.hdr[1] != 0) return;
  const int start = a.blk_start[(size_t)b * a.M + a.M - 1], len = a.blk_len[(size_t)b * a.M + a.M - 1];
  if (tok >= len) return;
  const float2 ml = lane < a.n_split ? a.part_ml[w * a.n_split + lane] : make_float2(-INFINITY, 0.f);
  float mx = ml.x;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  const float ref = (mx == -INFINITY) ? 0.f : mx;
  const float wgt = ml.y > 0.f ? exp2f(ml.x - ref) : 0.f;  // chunks that saw no key carry no output
  float l = ml.y * wgt;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) l += __shfl_xor_sync(0xffffffffu, l, off);
  const int sub = lane / (HD / 4), col = (lane % (HD / 4)) * 4;
  const float* const part = a.part_o + w * a.n_split * HD + col;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int c0 = 0; c0 < a.n_split; c0 += 4 * kSplit) {
    float4 o[4];
    float f[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = c0 + i * kSplit + sub;
      f[i] = __shfl_sync(0xffffffffu, wgt, c & 31);
      if (c >= a.n_split) f[i] = 0.f;
      o[i] = f[i] > 0.f ? load4(part + (int64_t)c * HD) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      acc.x = fmaf(o[i].x, f[i], acc.x); acc.y = fmaf(o[i].y, f[i], acc.y);
      acc.z = fmaf(o[i].z, f[i], acc.z); acc.w = fmaf(o[i].w, f[i], acc.w);
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

template <typename T, int HD>
int attn_combine_launch(const CombineArgs& c, cudaStream_t st) {
  const int64_t warps = (int64_t)c.B * c.N * c.lq_max;
  return launch_dependent(attn_combine_kernel<T, HD>, dim3((unsigned)((warps + 3) / 4)), dim3(128), 0, st, c);
}

}  // namespace brk
