// Shared helpers for the blockrank_b200 kernels (sm_100a only).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include <atomic>

#include "../../include/blockrank_b200.h"

namespace brk {

void set_error(const char* fmt, ...);

#define BRK_REQUIRE(cond, code, ...)  \
  do {                                \
    if (!(cond)) {                    \
      ::brk::set_error(__VA_ARGS__);  \
      return (code);                  \
    }                                 \
  } while (0)

#define BRK_CUDA(expr)                                                             \
  do {                                                                             \
    cudaError_t e_ = (expr);                                                       \
    if (e_ != cudaSuccess) {                                                       \
      ::brk::set_error("%s failed: %s", #expr, cudaGetErrorString(e_));            \
      return BRK_E_CUDA;                                                           \
    }                                                                              \
  } while (0)

// Kernels enqueued by this process; every launch below counts itself.
extern std::atomic<int64_t> g_launches;
// behind a <<<>>> launch
#define BRK_LAUNCHED()                                                             \
  do {                                                                             \
    BRK_CUDA(cudaGetLastError());                                                  \
    ::brk::g_launches.fetch_add(1, std::memory_order_relaxed);                     \
  } while (0)

// ---- element access helpers -------------------------------------------------
template <typename T>
struct Elem;
template <>
struct Elem<float> {
  static __device__ __forceinline__ float load(const float* p) { return *p; }
  static __device__ __forceinline__ void store(float* p, float v) { *p = v; }
  static __device__ __forceinline__ float round(float v) { return v; }
};
template <>
struct Elem<__nv_bfloat16> {
  static __device__ __forceinline__ float load(const __nv_bfloat16* p) { return __bfloat162float(*p); }
  static __device__ __forceinline__ void store(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }
  static __device__ __forceinline__ float round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
};

// 4 consecutive elements -> float4 (pointer must be aligned to 4 elements)
__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
  uint2 u = *reinterpret_cast<const uint2*>(p);
  __nv_bfloat162 a = *reinterpret_cast<__nv_bfloat162*>(&u.x);
  __nv_bfloat162 b = *reinterpret_cast<__nv_bfloat162*>(&u.y);
  float2 fa = __bfloat1622float2(a), fb = __bfloat1622float2(b);
  return make_float4(fa.x, fa.y, fb.x, fb.y);
}
__device__ __forceinline__ void store4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void store4(__nv_bfloat16* p, float4 v) {
  __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y);
  __nv_bfloat162 b = __floats2bfloat162_rn(v.z, v.w);
  uint2 u;
  u.x = *reinterpret_cast<uint32_t*>(&a);
  u.y = *reinterpret_cast<uint32_t*>(&b);
  *reinterpret_cast<uint2*>(p) = u;
}

// 8 consecutive elements <-> float[8] (pointer aligned to 8 elements)
__device__ __forceinline__ void load8(const float* p, float (&v)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&v)[8]) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[i]));
    v[2 * i] = f.x; v[2 * i + 1] = f.y;
  }
}
__device__ __forceinline__ void store8(float* p, const float (&v)[8]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float (&v)[8]) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    w[i] = *reinterpret_cast<uint32_t*>(&h);
  }
  *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
}

// Launch that may start before the preceding kernel of the stream has finished (its blocks become resident while that one
// drains); the kernel must execute ptx::grid_dependency_wait() before it touches memory.
// `cluster` neighbouring blocks (in x, a divisor of the grid) form a cluster.
template <typename K, typename... A>
int launch_dependent_clusters(int cluster, K kernel, dim3 grid, dim3 block, size_t smem, cudaStream_t st, const A&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2] = {};
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = cluster;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  BRK_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return BRK_OK;
}
template <typename K, typename... A>
int launch_dependent(K kernel, dim3 grid, dim3 block, size_t smem, cudaStream_t st, const A&... args) {
  return launch_dependent_clusters(1, kernel, grid, block, smem, st, args...);
}

struct View {
  char* ptr;
  int64_t sb, sh, ss;
};
inline View make_view(const brk_view& v) { return View{(char*)v.ptr, v.stride_b, v.stride_h, v.stride_s}; }

// Every attention call gets a 256-byte header at the start of its workspace: [0] the work counter of the
// tensor-core kernel, [1] the verdict of the span check (non-zero: malformed, the kernels write nothing).
constexpr size_t kWsHeader = 256;
// Values of the caller's status word: 10..49 (forward) and 60..80 (backward) name the bounded wait that gave up first in its thread
// (10..19 TMA warp, 20..29 MMA warps, 34, 35, 38, 39 output warps, other 30..39 softmax warps, 40, 41 one of the last three at
// the job ring; even numbers chain 0, odd ones chain 1), 50 malformed block spans, 51 a signal row outside the prompt, 90 the
// self-test's wait, 91 a self-test that found something else.
constexpr int kStatusBadSpans = 50;
constexpr int kStatusBadRows = 51;
constexpr int kStatusSelfTest = 90;

// kernel launchers implemented in the .cu files
int attn_prologue_launch(const brk_attn_params& p, int* hdr, float2* ml, int64_t n_ml, int4* win, int* n_live, int win_pitch,
                         cudaStream_t st);
int attn_simt_launch(const brk_attn_params& p, void* ws, size_t ws_bytes, cudaStream_t st);
int selftest_wait_launch(int32_t* status, uint32_t budget, cudaStream_t st);
int attn_tc_launch(const brk_attn_params& p, void* ws, size_t ws_bytes, cudaStream_t st);
size_t attn_f32_workspace(const brk_attn_params& p);
int attn_f32_launch(const brk_attn_params& p, void* ws, size_t ws_bytes, cudaStream_t st);
// bound on the last block's length
inline int query_rows(const brk_attn_params& p) {
  return (p.max_query_len > 0 && p.max_query_len < p.max_block_len) ? p.max_query_len : p.max_block_len;
}
// Key chunks whose partial results (fp32 rows of the output, max and sum) stay within 512 MB: a query block long enough to exceed
// that has row tiles for every SM without being cut (two blocks of 32,768 slots, fp32: 17 GB of partials in 32 chunks).
inline int capped_chunks(const brk_attn_params& p, int n) {
  const size_t chunk = (size_t)p.B * p.N * query_rows(p) * (p.D * sizeof(float) + sizeof(float2));
  return n > 1 && chunk * n > (512u << 20) ? (int)((512u << 20) / chunk > 1 ? (512u << 20) / chunk : 1) : n;
}
size_t attn_tc_workspace(const brk_attn_params& p);
size_t attn_bwd_workspace(const brk_attn_bwd_params& p);
int attn_bwd_launch(const brk_attn_bwd_params& p, void* ws, size_t ws_bytes, int32_t* status, cudaStream_t st);
int attn_bwd_f32_launch(const brk_attn_bwd_params& p, float* delta, cudaStream_t st);
bool attn_bwd_tc_supported(const brk_attn_bwd_params& p);
size_t attn_bwd_tc_extra_bytes(const brk_attn_bwd_params& p);
int attn_bwd_tc_launch(const brk_attn_bwd_params& p, float* delta, float* ws32, float* dq32, void* extra, int32_t* status,
                       cudaStream_t st);
int attn_bwd_mma_launch(const brk_attn_bwd_params& p, float* delta, float* dk32, float* dv32, float* dq32, cudaStream_t st);
int sm_count();

}  // namespace brk

namespace brk {
size_t doc_scores_workspace(const brk_score_params& p);
int doc_scores_launch(const brk_score_params& p, void* ws, size_t ws_bytes, cudaStream_t st);
int raw_scores_launch(const brk_score_params& p, void* out, cudaStream_t st);
size_t raw_scores_bwd_workspace(const brk_score_params& p);
int raw_scores_bwd_launch(const brk_score_params& p, const void* d_raw, const brk_view& dq, const brk_view& dk,
                          int accumulate, void* ws, size_t ws_bytes, cudaStream_t st);
int doc_scores_static_launch(const brk_score_params& p, cudaStream_t st);
int spans_launch(const uint8_t* mask, int B, int M, int H, int32_t* start, int32_t* len, cudaStream_t st);
int rmsnorm_launch(int dtype, const void* x, void* residual, const void* w, void* out, int64_t rows, int hidden,
                   float eps, cudaStream_t st);
int rope_launch(int dtype, void* q, int64_t q_rs, int N, void* k, int64_t k_rs, int Nk, int D, const int32_t* pos,
                const float* inv_freq, int64_t T, cudaStream_t st);
constexpr int kRankPackDocs = BRK_RANK_PACK_DOCS;
int rank_pack_launch(const float* logits, int B, int nd, int k, float* out, int64_t* top, const int32_t* status,
                     int32_t* status_out, cudaStream_t st);
int signal_rows_launch(const void* x, int row_bytes, const int32_t* pos, const int32_t* rows, int B, int S, int R, void* x_out,
                       int32_t* pos_out, int32_t* local, int32_t* status, cudaStream_t st);
int silu_mul_launch(int dtype, const void* gu, void* out, int64_t rows, int inter, cudaStream_t st);
}  // namespace brk
