// Warp-level bf16 tensor-core building blocks (mma.sync m16n8k16, ldmatrix, cp.async) shared by the kernels whose
// products are too skinny for a tcgen05 tile, and by the backward of blocks too long for the tcgen05 backward.
#pragma once
#include "brk_common.cuh"

namespace brk {

__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], const void* p) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(s));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], const void* p) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(s));
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_bf16(float x, float y) {
  __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
  return *reinterpret_cast<uint32_t*>(&h);
}

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async16_zfill(void* smem_dst, const void* gmem_src, bool valid) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem_dst);
  const int n = valid ? 16 : 0;  // 0 source bytes: the 16 destination bytes are filled with zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(gmem_src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async4(void* smem_dst, const void* gmem_src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

constexpr int kMmaTileRows = 64;  // tokens (rows or keys) per staged tile
template <int D>
struct MmaTile {
  static constexpr int kPitch = D + 8;  // elements: 16 bytes of padding per row
  __nv_bfloat16 e[kMmaTileRows][kPitch];
};

// acc[16 x D] += A[16 x 16] * Z[k0 .. k0+16][0 .. D)   (acc[nt] covers columns [8 nt, 8 nt + 8))
template <int D>
__device__ __forceinline__ void mm_nn_acc(float (&acc)[D / 8][4], const uint32_t (&a)[4], const MmaTile<D>& z, int k0, int lane) {
  const int j = lane >> 3, r = lane & 7;
#pragma unroll
  for (int np = 0; np < D / 16; ++np) {
    uint32_t bfr[4];
    ldsm_x4_t(bfr, &z.e[k0 + r + (j & 1) * 8][np * 16 + (j >> 1) * 8]);
    mma16816(acc[2 * np], a, bfr[0], bfr[1]);
    mma16816(acc[2 * np + 1], a, bfr[2], bfr[3]);
  }
}

}  // namespace brk
