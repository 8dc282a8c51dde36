// BlockRank attention forward for fp32 models on CUDA cores (tensor cores would drop to tf32).
//
// A CTA of 256 threads owns 64 query rows (64 / G consecutive tokens x the G heads of a KV head) of one block and walks
// through the list of keys those rows see -- the prefix block (documents) or every earlier slot (query block), then the
// own keys -- 64 at a time.  Both products are register-tiled: thread (ty, tx) keeps rows ty + 16 i of the scores (4 x 4,
// packed two head_dim elements per fma.rn.f32x2) and of the output (4 x D / 16).  The kernel is bound by the FMA pipe and
// by the latency in front of it: an inner step of 64 FMAs reads 8 16-byte pieces of shared memory, 12 wavefronts per warp.
// Two CTAs share an SM (101 KB each), so one computes while the other loads or exponentiates.  (Tiles of 8 x 4 need fewer
// wavefronts per FMA but leave two warps per scheduler: 399 us where this took 351.)
//
// The query block's context is cut into chunks of about 512 keys whose partial results attn_combine_kernel merges: its
// rows see thousands of keys where a document's see a few hundred, and as single CTAs they were the tail of the launch.
//
// One prompt of 20 documents (32/8 heads, head_dim 128, 8.4 GFLOP visible): 360 us (351 with one sum over head_dim); one query row per four threads with
// the keys re-read from shared memory for every row took 1,790 us.
#include <algorithm>

#include "attn_combine.cuh"
#include "brk_common.cuh"
#include "mma_bf16.cuh"
#include "tc_ptx.cuh"

namespace brk {

namespace {

constexpr int kThreads = 256;
constexpr int kRowStep = kThreads / 16, kR = 64 / kRowStep;  // a thread's rows: ty + kRowStep i, i < kR
constexpr int kRows = 64;
constexpr int kKeys = 64;
constexpr int kChunkKeys = 512;  // context keys of one chunk of the query block, about
constexpr int kMaxChunks = 32;
constexpr int kPitchP = 80;      // probabilities: the two rows of a warp's store fall on different banks

struct F32Args {
  View q, k, v, o;
  float* lse;
  const int32_t* blk_start;
  const int32_t* blk_len;
  const int* hdr;  // [1] != 0: the prologue kernel found the block spans malformed
  int B, N, Nk, S, M, G;
  int lq, q_tiles, n_chunk;  // query block: rows per head of the partial buffers, row tiles, chunks
  int tiles;                 // row tiles of any other block
  int n_query;               // CTAs of the query blocks; the rest are the other blocks'
  float scale_log2;
  float* part_o;    // [B, N, lq, n_chunk, D]
  float2* part_ml;  // [B, N, lq, n_chunk]
};

__device__ __forceinline__ bool slot_valid(const int32_t* bs, const int32_t* bl, int M, int s) {
  int lo = 0, hi = M;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (bs[mid] <= s) lo = mid + 1; else hi = mid;
  }
  const int m = lo - 1;
  return m >= 0 && s < bs[m] + bl[m];
}

template <int D>
__global__ void __launch_bounds__(kThreads, 2) attn_f32_kernel(F32Args a) {
  constexpr int kPitch = D + 4;
  constexpr int kE = D / 16;  // output elements per thread and row: tx * 4 + {0..3} (+ 64)
  extern __shared__ __align__(16) float fsm[];
  float* const qs = fsm;                      // [64][kPitch], scaled
  float* const ks = qs + kRows * kPitch;      // [64][kPitch]; the probabilities [64][kPitchP] once the scores are taken
  constexpr int kKsFloats = kKeys * (kPitch > kPitchP ? kPitch : kPitchP);
  float* const vs = ks + kKsFloats;           // [64][D]
  __shared__ int s_slot[kKeys];               // slot of each key of the tile, -1: none
  ptx::grid_dependency_wait();
  if (a.hdr[1] != 0) return;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const bool query = (int)blockIdx.x < a.n_query;
  int b, g, m, tile, chunk = 0;
  {
    int x = query ? blockIdx.x : blockIdx.x - a.n_query;
    const int per = query ? a.q_tiles * a.n_chunk : (a.M - 1) * a.tiles;
    const int bg = x / per;
    x %= per;
    b = bg / a.Nk;
    g = bg % a.Nk;
    if (query) {
      m = a.M - 1;
      tile = x / a.n_chunk;
      chunk = x % a.n_chunk;
    } else {
      m = x / a.tiles;
      tile = x % a.tiles;
    }
  }
  const int32_t* bs = a.blk_start + (size_t)b * a.M;
  const int32_t* bl = a.blk_len + (size_t)b * a.M;
  const int start = bs[m], len = bl[m], G = a.G, TQ = kRows / G;
  float* const ob = reinterpret_cast<float*>(a.o.ptr) + (int64_t)b * a.o.sb;
  {
    // Padding slots are zero: the gap in front of a block by its first CTA, the one behind the last block in slices.
    const int per_row = G * (D / 4);
    auto zero_rows = [&](int lo, int hi) {
      for (int i = tid; i < (hi - lo) * per_row; i += kThreads) {
        const int s = lo + i / per_row, rem = i % per_row;
        store4(ob + (int64_t)s * a.o.ss + (int64_t)(g * G + rem / (D / 4)) * a.o.sh + rem % (D / 4) * 4, make_float4(0.f, 0.f, 0.f, 0.f));
      }
    };
    if (tile == 0 && chunk == 0) zero_rows(m == 0 ? 0 : bs[m - 1] + bl[m - 1], start);
    if (query) {
      const int lo = start + len, rows = a.S - lo, parts = a.q_tiles * a.n_chunk, mine = tile * a.n_chunk + chunk;
      const int per = (rows + parts - 1) / parts;
      if (rows > 0) zero_rows(lo + min(rows, mine * per), lo + min(rows, (mine + 1) * per));
    }
  }
  const int t0 = tile * TQ;
  if (t0 >= len) return;

  // the key list: context slots [ctx_lo, ctx_lo + n_ctx), then own keys up to this tile's last token
  int ctx_lo = 0, n_ctx = 0;
  if (m > 0) {
    ctx_lo = bs[0];
    n_ctx = query ? bs[m - 1] + bl[m - 1] - ctx_lo : bl[0];
  }
  int j_lo = 0, j_hi = n_ctx + min(len, t0 + TQ);
  if (query && a.n_chunk > 1) {
    const int per = ((n_ctx + a.n_chunk - 1) / a.n_chunk + kKeys - 1) / kKeys * kKeys;
    j_lo = min(n_ctx, chunk * per);
    if (chunk + 1 < a.n_chunk) j_hi = min(n_ctx, j_lo + per);
  }
  const bool gaps = query && m > 0;  // the context range may contain padding slots

  for (int i = tid; i < kRows * (D / 4); i += kThreads) {
    const int r = i / (D / 4), d = i % (D / 4) * 4, tok = min(t0 + r / G, len - 1);
    const float4 x = load4(reinterpret_cast<const float*>(a.q.ptr) + (int64_t)b * a.q.sb + (int64_t)(g * G + r % G) * a.q.sh +
                           (int64_t)(start + tok) * a.q.ss + d);
    store4(qs + r * kPitch + d, make_float4(x.x * a.scale_log2, x.y * a.scale_log2, x.z * a.scale_log2, x.w * a.scale_log2));
  }
  float m_run[kR], l_run[kR];
  ptx::f32x2 o[kR][kE / 2];
#pragma unroll
  for (int i = 0; i < kR; ++i) {
    m_run[i] = -INFINITY;
    l_run[i] = 0.f;
#pragma unroll
    for (int e = 0; e < kE / 2; ++e) o[i][e] = 0ull;
  }
  const float* const kb = reinterpret_cast<const float*>(a.k.ptr) + (int64_t)b * a.k.sb + (int64_t)g * a.k.sh;
  const float* const vb = reinterpret_cast<const float*>(a.v.ptr) + (int64_t)b * a.v.sb + (int64_t)g * a.v.sh;

  for (int j0 = j_lo; j0 < j_hi; j0 += kKeys) {
    __syncthreads();  // the previous tile's probabilities and values have been read
    bool any = false;
    if (tid < kKeys) {
      const int j = j0 + tid;
      int slot = -1;
      if (j < j_hi) {
        slot = j < n_ctx ? ctx_lo + j : start + j - n_ctx;
        if (gaps && j < n_ctx && !slot_valid(bs, bl, a.M, slot)) slot = -1;
      }
      s_slot[tid] = slot;
      any = slot >= 0;
    }
    if (!__syncthreads_or(any)) continue;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const float* const src = half ? vb : kb;
      const int64_t stride = half ? a.v.ss : a.k.ss;
      for (int i = tid; i < kKeys * (D / 4); i += kThreads) {
        const int r = i / (D / 4), d = i % (D / 4) * 4, slot = s_slot[r];
        cp_async16_zfill(half ? vs + r * D + d : ks + r * kPitch + d, src + (int64_t)max(slot, 0) * stride + d, slot >= 0);
      }
      cp_async_commit();
    }
    cp_async_wait<1>();
    __syncthreads();
    // scores: rows ty + 16 i, keys tx + 16 c, in sums of 32 products (of 64 at head_dim 128, the output of short prompts was 5 %
    // further from 64 bits than the kernel before this one's)
    constexpr int kParts = D / 64;
    float s[kR][4];
#pragma unroll
    for (int h = 0; h < kParts; ++h) {
      ptx::f32x2 acc[kR][4];
#pragma unroll
      for (int i = 0; i < kR; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[i][c] = 0ull;
#pragma unroll 1
      for (int d = h * 64; d < (h + 1) * 64; d += 4) {
        ulonglong2 kk[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) kk[c] = *reinterpret_cast<const ulonglong2*>(ks + (tx + 16 * c) * kPitch + d);
#pragma unroll
        for (int i = 0; i < kR; ++i) {
          const ulonglong2 qq = *reinterpret_cast<const ulonglong2*>(qs + (ty + kRowStep * i) * kPitch + d);
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[i][c] = ptx::fma2(qq.y, kk[c].y, ptx::fma2(qq.x, kk[c].x, acc[i][c]));
        }
      }
#pragma unroll
      for (int i = 0; i < kR; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          float x, y;
          ptx::unpack2(acc[i][c], x, y);
          s[i][c] = h ? s[i][c] + (x + y) : x + y;
        }
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int key = tx + 16 * c, own = j0 + key - n_ctx;  // own > token: behind the diagonal
      const bool none = s_slot[key] < 0;
#pragma unroll
      for (int i = 0; i < kR; ++i)
        if (none || own > t0 + (ty + kRowStep * i) / G) s[i][c] = -INFINITY;
    }
    __syncthreads();  // every thread has read the keys: their place takes the probabilities
#pragma unroll
    for (int i = 0; i < kR; ++i) {
      float mx = fmaxf(fmaxf(s[i][0], s[i][1]), fmaxf(s[i][2], s[i][3]));
#pragma unroll
      for (int off = 8; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
      const float m_new = fmaxf(m_run[i], mx), ref = m_new == -INFINITY ? 0.f : m_new;
      const float corr = exp2f(m_run[i] - ref);
      m_run[i] = m_new;
      float sum = 0.f;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float p = exp2f(s[i][c] - ref);
        sum += p;
        ks[(ty + kRowStep * i) * kPitchP + tx + 16 * c] = p;
      }
      l_run[i] = l_run[i] * corr + sum;  // (this thread's keys only: added up over the row at the end)
      const ptx::f32x2 c2 = ptx::pack2(corr, corr);
#pragma unroll
      for (int e = 0; e < kE / 2; ++e) o[i][e] = ptx::mul2(o[i][e], c2);
    }
    cp_async_wait<0>();
    __syncthreads();
    const int n4 = (min(kKeys, j_hi - j0) + 3) >> 2;
#pragma unroll 1
    for (int k4 = 0; k4 < n4; ++k4) {
      float4 p[kR];
#pragma unroll
      for (int i = 0; i < kR; ++i) p[i] = load4(ks + (ty + kRowStep * i) * kPitchP + k4 * 4);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        ulonglong2 v[kE / 4];
#pragma unroll
        for (int e = 0; e < kE / 4; ++e) v[e] = *reinterpret_cast<const ulonglong2*>(vs + (k4 * 4 + kk) * D + tx * 4 + e * 64);
#pragma unroll
        for (int i = 0; i < kR; ++i) {
          const float x = kk == 0 ? p[i].x : kk == 1 ? p[i].y : kk == 2 ? p[i].z : p[i].w;
          const ptx::f32x2 p2 = ptx::pack2(x, x);
#pragma unroll
          for (int e = 0; e < kE / 4; ++e) {
            o[i][2 * e] = ptx::fma2(p2, v[e].x, o[i][2 * e]);
            o[i][2 * e + 1] = ptx::fma2(p2, v[e].y, o[i][2 * e + 1]);
          }
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kR; ++i) {
    float l = l_run[i];
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) l += __shfl_xor_sync(0xffffffffu, l, off);
    const int r = ty + kRowStep * i, tok = t0 + r / G, n = g * G + r % G;
    if (tok >= len) continue;
    const bool part = query && a.n_chunk > 1;
    const float inv = part ? 1.f : l > 0.f ? 1.f / l : 0.f;
    const int64_t prow = (((int64_t)b * a.N + n) * a.lq + tok) * a.n_chunk + chunk;
    float* const dst = part ? a.part_o + prow * D : ob + (int64_t)(start + tok) * a.o.ss + (int64_t)n * a.o.sh;
#pragma unroll
    for (int e = 0; e < kE / 4; ++e) {
      float x, y, z, w;
      ptx::unpack2(o[i][2 * e], x, y);
      ptx::unpack2(o[i][2 * e + 1], z, w);
      store4(dst + tx * 4 + e * 64, make_float4(x * inv, y * inv, z * inv, w * inv));
    }
    if (tx == 0) {
      if (part) a.part_ml[prow] = make_float2(m_run[i], l);
      else if (a.lse) a.lse[((int64_t)b * a.N + n) * a.S + start + tok] = (m_run[i] + log2f(l)) * 0.6931471805599453f;
    }
  }
}

int chunks(const brk_attn_params& p) {
  return p.M < 2 ? 1 : capped_chunks(p, std::max(1, std::min(kMaxChunks, (p.S + kChunkKeys - 1) / kChunkKeys)));
}

template <int D>
int launch(const brk_attn_params& p, const F32Args& a, cudaStream_t st) {
  constexpr int kPitch = D + 4;
  constexpr int smem = (kRows * kPitch + kKeys * (kPitch > kPitchP ? kPitch : kPitchP) + kKeys * D) * (int)sizeof(float);
  BRK_CUDA(cudaFuncSetAttribute(attn_f32_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const int64_t ctas = a.n_query + (int64_t)p.B * p.Nk * (p.M - 1) * a.tiles;
  BRK_REQUIRE(ctas < (1ll << 31), BRK_E_UNSUPPORTED, "grid too large: B*Nk=%d M=%d", p.B * p.Nk, p.M);
  const int rc = launch_dependent(attn_f32_kernel<D>, dim3((unsigned)ctas), dim3(kThreads), smem, st, a);
  if (rc || a.n_chunk == 1) return rc;
  CombineArgs c{a.o, a.lse, a.blk_start, a.blk_len, a.hdr, p.B, p.N, p.S, p.M, a.lq, a.n_chunk, a.part_o, a.part_ml};
  return attn_combine_launch<float, D>(c, st);
}

}  // namespace

size_t attn_f32_workspace(const brk_attn_params& p) {
  const int nc = chunks(p);
  const size_t rows = (size_t)p.B * p.N * query_rows(p) * nc;
  return kWsHeader + (nc > 1 ? rows * (p.D * sizeof(float) + sizeof(float2)) : 0);
}

int attn_f32_launch(const brk_attn_params& p, void* ws, size_t ws_bytes, cudaStream_t st) {
  BRK_REQUIRE(ws != nullptr && ws_bytes >= attn_f32_workspace(p) && ((uintptr_t)ws & 15) == 0, BRK_E_WORKSPACE,
              "attention workspace: %zu bytes (16-byte aligned) needed, %zu given", attn_f32_workspace(p), ws_bytes);
  const int G = p.N / p.Nk;
  BRK_REQUIRE(G == 1 || G == 2 || G == 4 || G == 8, BRK_E_UNSUPPORTED, "SIMT attention supports N/Nk in {1,2,4,8}, got %d", G);
  F32Args a;
  a.q = make_view(p.q); a.k = make_view(p.k); a.v = make_view(p.v); a.o = make_view(p.o);
  a.lse = p.lse;
  a.blk_start = p.blk_start; a.blk_len = p.blk_len;
  a.hdr = reinterpret_cast<const int*>(ws);
  a.B = p.B; a.N = p.N; a.Nk = p.Nk; a.S = p.S; a.M = p.M; a.G = G;
  a.lq = query_rows(p);
  a.n_chunk = chunks(p);
  a.q_tiles = (int)(((int64_t)a.lq * G + kRows - 1) / kRows);
  a.tiles = (int)(((int64_t)p.max_block_len * G + kRows - 1) / kRows);
  const int64_t nq = (int64_t)p.B * p.Nk * a.q_tiles * a.n_chunk;
  BRK_REQUIRE(nq < (1ll << 30), BRK_E_UNSUPPORTED, "grid too large: B*Nk=%d M=%d", p.B * p.Nk, p.M);
  a.n_query = (int)nq;
  a.scale_log2 = p.scale * 1.4426950408889634f;
  const size_t rows = (size_t)p.B * p.N * a.lq * a.n_chunk;
  a.part_o = reinterpret_cast<float*>(static_cast<unsigned char*>(ws) + kWsHeader);
  a.part_ml = reinterpret_cast<float2*>(a.part_o + rows * p.D);
  // every (row, chunk) pair is written by the kernel, also of chunks without keys: nothing to reset
  int rc = attn_prologue_launch(p, reinterpret_cast<int*>(ws), nullptr, 0, nullptr, nullptr, 0, st);
  if (rc) return rc;
  if (p.D == 128) return launch<128>(p, a, st);
  if (p.D == 64) return launch<64>(p, a, st);
  set_error("SIMT attention supports head_dim 64 or 128, got %d", p.D);
  return BRK_E_UNSUPPORTED;
}

}  // namespace brk
