// BlockRank attention backward for fp32 models on CUDA cores.
//
// A CTA of 256 threads owns one tile of 64 keys of a block's key list -- for a document the prefix block's keys, then its
// own -- and walks through the row tiles (64 / G tokens x G heads) that see them: the block's own, then the query
// block's (which see the own keys).  With Q, dO, K, V tiles in shared memory all five products are register-tiled:
//   S = Q K^T, dP = dO V^T (4 x 4 per thread)   P = 2^(S - lse)   dS = P (dP - delta)
//   dV += P^T dO, dK += dS^T Q (4 keys x D / 16 per thread, in registers over all row tiles)   dQ = dS K
// dQ, and dK / dV of the prefix (which every document's rows see), are added into the zeroed outputs with fp32 vector
// reductions, in no fixed order: rows seen by more than two key tiles, and the prefix, can differ in the last bits from call
// to call.  dK / dV of own keys are stored.  Bound by the FMA pipe: 2.6 MFMA per (key tile, row tile) pair for 64 KB of loads;
// fma.rn.f32x2 keeps the issue slots free for the shared-memory reads.
//
// One prompt of 20 documents of 120..160 tokens (32/8 heads, head_dim 128): 926 us; one row or key per four threads, in two
// kernels, took 3,530.
#include <algorithm>

#include "brk_common.cuh"
#include "mma_bf16.cuh"
#include "tc_ptx.cuh"

namespace brk {

namespace {

constexpr int kThreads = 256;
constexpr int kTile = 64;
constexpr int kPitchS = kTile + 4;

struct BwdF32Args {
  View q, k, v, o, d_o, dq, dk, dv;
  const float* lse;
  float* delta;  // [B, N, S]
  const int32_t* blk_start;
  const int32_t* blk_len;
  int B, N, Nk, S, M, G, max_block_len, key_tiles;
  float scale, scale_log2;
};

__device__ __forceinline__ void span_of(const BwdF32Args& a, int b, int m, int& start, int& len) {
  start = a.blk_start[(size_t)b * a.M + m];
  len = a.blk_len[(size_t)b * a.M + m];
  if (start < 0 || len < 0 || len > a.max_block_len || start > a.S - len) len = 0;  // skipped: nothing out of bounds
}

__device__ __forceinline__ void red4(float* p, float x, float y, float z, float w) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}
__device__ __forceinline__ void red4(float* p, ptx::f32x2 lo, ptx::f32x2 hi, float f) {
  float x, y, z, w;
  ptx::unpack2(lo, x, y);
  ptx::unpack2(hi, z, w);
  red4(p, x * f, y * f, z * f, w * f);
}

// delta = rowsum(dO * O), one warp per (prompt, slot, head); and zeros in dq, dk, dv.
__global__ void __launch_bounds__(256) attn_bwd_f32_prep_kernel(BwdF32Args a, int D) {
  const int64_t w = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (w >= (int64_t)a.B * a.S * a.N) return;
  const int n = (int)(w % a.N), s = (int)(w / a.N % a.S), b = (int)(w / ((int64_t)a.N * a.S));
  auto row = [&](const View& t) { return reinterpret_cast<float*>(t.ptr) + (int64_t)b * t.sb + (int64_t)n * t.sh + (int64_t)s * t.ss + lane * 4; };
  float d = 0.f;
  if (lane * 4 < D) {
    const float4 x = load4(row(a.d_o)), y = load4(row(a.o));
    d = x.x * y.x + x.y * y.y + x.z * y.z + x.w * y.w;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    store4(row(a.dq), zero);
    if (n < a.Nk) {
      store4(row(a.dk), zero);
      store4(row(a.dv), zero);
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) d += __shfl_xor_sync(0xffffffffu, d, off);
  if (lane == 0) a.delta[((size_t)b * a.N + n) * a.S + s] = d;
}

// sum[i][e] += sum over r of w[r][4 ty + i] x[r][own dims]: 4 keys x D / 16 elements per thread, w [64][kPitchS].  The tile's
// rows are summed among themselves first: with hundreds of them added one by one to the running sums, dK and dV were up to a
// quarter further from 64 bits (8 heads on one KV head, head_dim 64, 20 documents: 8.0e-7, now 3.5e-7).
template <int D>
__device__ __forceinline__ void tn_acc(ptx::f32x2 (&sum)[4][D / 32], const float* w, const float* x, int rows, int ty, int tx) {
  ptx::f32x2 acc[4][D / 32];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int e = 0; e < D / 32; ++e) acc[i][e] = 0ull;
#pragma unroll 2
  for (int r = 0; r < rows; ++r) {
    const float4 p = load4(w + r * kPitchS + ty * 4);
    const ptx::f32x2 p2[4] = {ptx::pack2(p.x, p.x), ptx::pack2(p.y, p.y), ptx::pack2(p.z, p.z), ptx::pack2(p.w, p.w)};
#pragma unroll
    for (int e = 0; e < D / 64; ++e) {
      const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(x + r * (D + 4) + tx * 4 + e * 64);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        acc[i][2 * e] = ptx::fma2(p2[i], v.x, acc[i][2 * e]);
        acc[i][2 * e + 1] = ptx::fma2(p2[i], v.y, acc[i][2 * e + 1]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int e = 0; e < D / 32; ++e) sum[i][e] = ptx::add2(sum[i][e], acc[i][e]);
}

// c[i][j] = x[ty + 16 i] . y[tx + 16 j] over D, in four sums of D / 4 (one long one leaves every probability further from 64
// bits)
template <int D>
__device__ __forceinline__ void nt(float (&c)[4][4], const float* x, const float* y, int ty, int tx) {
  ptx::f32x2 acc[4][4], first[4][4];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (h) first[i][j] = acc[i][j];
        acc[i][j] = 0ull;
      }
#pragma unroll 4
    for (int d = h * (D / 2); d < (h + 1) * (D / 2); d += 4) {
      ulonglong2 yy[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) yy[j] = *reinterpret_cast<const ulonglong2*>(y + (tx + 16 * j) * (D + 4) + d);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const ulonglong2 xx = *reinterpret_cast<const ulonglong2*>(x + (ty + 16 * i) * (D + 4) + d);
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = ptx::fma2(xx.y, yy[j].y, ptx::fma2(xx.x, yy[j].x, acc[i][j]));
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float lo, hi;
      ptx::unpack2(ptx::add2(first[i][j], acc[i][j]), lo, hi);
      c[i][j] = lo + hi;
    }
}

template <int D>
__global__ void __launch_bounds__(kThreads, 1) attn_bwd_f32_kernel(BwdF32Args a) {
  constexpr int kPitch = D + 4;
  extern __shared__ __align__(16) float fsm[];
  float* const ks = fsm;
  float* const vs = ks + kTile * kPitch;
  float* const qs = vs + kTile * kPitch;
  float* const gs = qs + kTile * kPitch;
  float* const ps = gs + kTile * kPitch;
  float* const ds = ps + kTile * kPitchS;
  __shared__ float s_lse[kTile], s_delta[kTile];
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15, G = a.G, TQ = kTile / G;
  const int kt = blockIdx.x % a.key_tiles, m = blockIdx.x / a.key_tiles, b = blockIdx.y / a.Nk, g = blockIdx.y % a.Nk;
  int start, len, s0 = 0, l0 = 0, qstart = 0, ql = 0;
  span_of(a, b, m, start, len);
  if (m > 0 && m < a.M - 1) span_of(a, b, 0, s0, l0);
  if (m < a.M - 1) span_of(a, b, a.M - 1, qstart, ql);
  const int k0 = kt * kTile;
  if (len == 0 || k0 >= l0 + len) return;
  const float* const kb = reinterpret_cast<const float*>(a.k.ptr) + (int64_t)b * a.k.sb + (int64_t)g * a.k.sh;
  const float* const vb = reinterpret_cast<const float*>(a.v.ptr) + (int64_t)b * a.v.sb + (int64_t)g * a.v.sh;
  const int nkey = min(kTile, l0 + len - k0);
  auto key_slot = [&](int j) { return j < l0 ? s0 + j : start + j - l0; };
  for (int i = tid; i < kTile * (D / 4); i += kThreads) {
    const int r = i / (D / 4), d = i % (D / 4) * 4, slot = key_slot(k0 + min(r, nkey - 1));
    cp_async16_zfill(ks + r * kPitch + d, kb + (int64_t)slot * a.k.ss + d, r < nkey);
    cp_async16_zfill(vs + r * kPitch + d, vb + (int64_t)slot * a.v.ss + d, r < nkey);
  }
  ptx::f32x2 dk[4][D / 32], dv[4][D / 32];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int e = 0; e < D / 32; ++e) dk[i][e] = dv[i][e] = 0ull;
  const int r0 = max(0, k0 - l0) / TQ, n_own = (len + TQ - 1) / TQ - r0;
  const int n_rows = n_own + (k0 + kTile > l0 ? (ql + TQ - 1) / TQ : 0);
  for (int it = 0; it < n_rows; ++it) {
    const bool own = it < n_own;
    const int t0 = (own ? r0 + it : it - n_own) * TQ, first = (own ? start : qstart) + t0;
    const int nrow = min(kTile, ((own ? len : ql) - t0) * G);
    __syncthreads();  // the previous tile has been read
    for (int i = tid; i < kTile * (D / 4); i += kThreads) {
      const int r = i / (D / 4), d = i % (D / 4) * 4, rr = min(r, nrow - 1), slot = first + rr / G, n = g * G + rr % G;
      cp_async16_zfill(qs + r * kPitch + d, reinterpret_cast<const float*>(a.q.ptr) + (int64_t)b * a.q.sb + (int64_t)n * a.q.sh + (int64_t)slot * a.q.ss + d, r < nrow);
      cp_async16_zfill(gs + r * kPitch + d, reinterpret_cast<const float*>(a.d_o.ptr) + (int64_t)b * a.d_o.sb + (int64_t)n * a.d_o.sh + (int64_t)slot * a.d_o.ss + d, r < nrow);
    }
    if (tid < kTile) {
      float l = INFINITY, d = 0.f;  // rows beyond the block: P = 0
      if (tid < nrow) {
        const size_t id = ((size_t)b * a.N + g * G + tid % G) * a.S + first + tid / G;
        l = a.lse[id] * 1.4426950408889634f;
        d = a.delta[id];
      }
      s_lse[tid] = l;
      s_delta[tid] = d;
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    {
      float p[4][4], x[4][4];
      nt<D>(p, qs, ks, ty, tx);
      nt<D>(x, gs, vs, ty, tx);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = ty + 16 * i, tok = t0 + r / G;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int key = tx + 16 * j, pos = k0 + key - l0;  // < 0: prefix
          const bool vis = key < nkey && (own ? pos <= tok : pos >= 0);
          const float pv = vis ? exp2f(p[i][j] * a.scale_log2 - s_lse[r]) : 0.f;
          ps[r * kPitchS + key] = pv;
          ds[r * kPitchS + key] = pv * (x[i][j] - s_delta[r]);
        }
      }
    }
    __syncthreads();
    tn_acc<D>(dv, ps, gs, nrow, ty, tx);
    tn_acc<D>(dk, ds, qs, nrow, ty, tx);
    // dQ: rows ty + 16 i, own dims
    ptx::f32x2 dq[4][D / 32];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int e = 0; e < D / 32; ++e) dq[i][e] = 0ull;
#pragma unroll 1
    for (int c = 0; c < nkey; c += 4) {
      float4 w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) w[i] = load4(ds + (ty + 16 * i) * kPitchS + c);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
#pragma unroll
        for (int e = 0; e < D / 64; ++e) {
          const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(ks + (c + kk) * kPitch + tx * 4 + e * 64);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float f = kk == 0 ? w[i].x : kk == 1 ? w[i].y : kk == 2 ? w[i].z : w[i].w;
            const ptx::f32x2 f2 = ptx::pack2(f, f);
            dq[i][2 * e] = ptx::fma2(f2, y.x, dq[i][2 * e]);
            dq[i][2 * e + 1] = ptx::fma2(f2, y.y, dq[i][2 * e + 1]);
          }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = ty + 16 * i;
      if (r >= nrow) continue;
      float* const dst = reinterpret_cast<float*>(a.dq.ptr) + (int64_t)b * a.dq.sb + (int64_t)(g * G + r % G) * a.dq.sh +
                         (int64_t)(first + r / G) * a.dq.ss + tx * 4;
#pragma unroll
      for (int e = 0; e < D / 64; ++e) red4(dst + e * 64, dq[i][2 * e], dq[i][2 * e + 1], a.scale);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int j = k0 + ty * 4 + i;
    if (j >= l0 + len) continue;
    const int64_t slot = key_slot(j);
    float* const pk = reinterpret_cast<float*>(a.dk.ptr) + (int64_t)b * a.dk.sb + (int64_t)g * a.dk.sh + slot * a.dk.ss + tx * 4;
    float* const pv = reinterpret_cast<float*>(a.dv.ptr) + (int64_t)b * a.dv.sb + (int64_t)g * a.dv.sh + slot * a.dv.ss + tx * 4;
#pragma unroll
    for (int e = 0; e < D / 64; ++e) {
      if (j < l0 || m == 0) {  // the prefix: other items add to it
        red4(pk + e * 64, dk[i][2 * e], dk[i][2 * e + 1], a.scale);
        red4(pv + e * 64, dv[i][2 * e], dv[i][2 * e + 1], 1.f);
      } else {
        float x, y, z, w;
        ptx::unpack2(dk[i][2 * e], x, y);
        ptx::unpack2(dk[i][2 * e + 1], z, w);
        store4(pk + e * 64, make_float4(x * a.scale, y * a.scale, z * a.scale, w * a.scale));
        ptx::unpack2(dv[i][2 * e], x, y);
        ptx::unpack2(dv[i][2 * e + 1], z, w);
        store4(pv + e * 64, make_float4(x, y, z, w));
      }
    }
  }
}

template <int D>
int launch(const BwdF32Args& a, cudaStream_t st) {
  constexpr int smem = (4 * kTile * (D + 4) + 2 * kTile * kPitchS) * (int)sizeof(float);
  BRK_CUDA(cudaFuncSetAttribute(attn_bwd_f32_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  attn_bwd_f32_kernel<D><<<dim3((unsigned)(a.key_tiles * a.M), (unsigned)(a.B * a.Nk)), kThreads, smem, st>>>(a);
  BRK_LAUNCHED();
  return BRK_OK;
}

}  // namespace

int attn_bwd_f32_launch(const brk_attn_bwd_params& p, float* delta, cudaStream_t st) {
  BwdF32Args a;
  a.q = make_view(p.q); a.k = make_view(p.k); a.v = make_view(p.v); a.o = make_view(p.o); a.d_o = make_view(p.d_o);
  a.dq = make_view(p.dq); a.dk = make_view(p.dk); a.dv = make_view(p.dv);
  a.lse = p.lse;
  a.delta = delta;
  a.blk_start = p.blk_start; a.blk_len = p.blk_len;
  a.B = p.B; a.N = p.N; a.Nk = p.Nk; a.S = p.S; a.M = p.M; a.G = p.N / p.Nk; a.max_block_len = p.max_block_len;
  // longest key list: a document behind the prefix
  a.key_tiles = (int)(((int64_t)p.max_block_len * (p.M > 2 ? 2 : 1) + kTile - 1) / kTile);
  a.scale = p.scale;
  a.scale_log2 = p.scale * 1.4426950408889634f;
  const int64_t rows = (int64_t)p.B * p.S * p.N;
  BRK_REQUIRE(p.B * p.Nk <= 65535 && (int64_t)a.key_tiles * p.M < (1ll << 31) && (rows + 7) / 8 < (1ll << 31), BRK_E_UNSUPPORTED,
              "grid too large: B*Nk=%d M=%d", p.B * p.Nk, p.M);
  attn_bwd_f32_prep_kernel<<<(unsigned)((rows + 7) / 8), 256, 0, st>>>(a, p.D);
  BRK_LAUNCHED();
  return p.D == 128 ? launch<128>(a, st) : launch<64>(a, st);
}

}  // namespace brk
