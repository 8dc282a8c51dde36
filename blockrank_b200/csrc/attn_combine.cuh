// Merge of the query block's key chunks, shared by the tcgen05 and the fp32 attention kernels.
#pragma once
#include "brk_common.cuh"

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

// One warp per (prompt, head, query token).
template <typename T, int HD>
__global__ void __launch_bounds__(128) attn_combine_kernel(CombineArgs a) {
  if (a.hdr[1] != 0) return;
  const int lane = threadIdx.x & 31;
  const int64_t w = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  const int64_t total = (int64_t)a.B * a.N * a.lq_max;
  if (w >= total) return;
  const int tok = (int)(w % a.lq_max);
  const int n = (int)((w / a.lq_max) % a.N);
  const int b = (int)(w / ((int64_t)a.lq_max * a.N));
  const int start = a.blk_start[(size_t)b * a.M + a.M - 1], len = a.blk_len[(size_t)b * a.M + a.M - 1];
  if (tok >= len) return;
  const float2* ml = a.part_ml + w * a.n_split;
  const int col = (lane * 4) & (HD - 1);  // (head_dim 64: the upper half of the warp repeats the lower one's work)
  float mx = -INFINITY;
  for (int c = 0; c < a.n_split; ++c) mx = fmaxf(mx, ml[c].x);
  const float ref = (mx == -INFINITY) ? 0.f : mx;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  float l = 0.f;
  for (int c = 0; c < a.n_split; ++c) {
    const float2 x = ml[c];
    if (x.y > 0.f) {  // chunks that saw no key carry no output
      const float wgt = exp2f(x.x - ref);
      const float4 o = *reinterpret_cast<const float4*>(a.part_o + (w * a.n_split + c) * HD + col);
      acc.x = fmaf(o.x, wgt, acc.x); acc.y = fmaf(o.y, wgt, acc.y);
      acc.z = fmaf(o.z, wgt, acc.z); acc.w = fmaf(o.w, wgt, acc.w);
      l = fmaf(x.y, wgt, l);
    }
  }
  const float inv = l > 0.f ? 1.f / l : 0.f;
  T* dst = reinterpret_cast<T*>(a.o.ptr) + (int64_t)b * a.o.sb + (int64_t)(start + tok) * a.o.ss + (int64_t)n * a.o.sh + col;
  if (lane * 4 < HD) store4(dst, make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv));
  if (a.lse != nullptr && lane == 0) a.lse[((int64_t)b * a.N + n) * a.S + start + tok] = (ref + log2f(l)) * 0.6931471805599453f;
}

template <typename T, int HD>
int attn_combine_launch(const CombineArgs& c, cudaStream_t st) {
  const int64_t warps = (int64_t)c.B * c.N * c.lq_max;
  attn_combine_kernel<T, HD><<<(unsigned)((warps + 3) / 4), 128, 0, st>>>(c);
  BRK_CUDA(cudaGetLastError());
  return BRK_OK;
}

}  // namespace brk
