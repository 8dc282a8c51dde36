// Parameters shared by the document-score and raw-score kernels.
#pragma once
#include "brk_common.cuh"

namespace brk {

struct ScoreArgs {
  View q, k;
  const int32_t* rows;
  const int32_t* blk_start;
  const int32_t* blk_len;
  float2* partial;  // [B, N, R, nd]
  float* mass;      // [B, N, R, nd] out
  float* logits;    // [B, nd] out, optional
  float inv_count_temp;  // 1 / (N * R * temperature)
  int B, N, Nk, S, M, R;
  float scale;
};

inline ScoreArgs make_score_args(const brk_score_params& p) {
  ScoreArgs a;
  a.q = make_view(p.q);
  a.k = make_view(p.k);
  a.rows = p.rows;
  a.blk_start = p.blk_start;
  a.blk_len = p.blk_len;
  a.partial = nullptr;
  a.mass = nullptr;
  a.logits = nullptr;
  a.inv_count_temp = 0.f;
  a.B = p.B; a.N = p.N; a.Nk = p.Nk; a.S = p.S; a.M = p.M; a.R = p.R;
  a.scale = p.scale;
  return a;
}

inline int check_score_params(const brk_score_params& p) {
  BRK_REQUIRE(p.q.ptr && p.k.ptr && p.blk_start && p.blk_len, BRK_E_ARG, "null pointer in score params");
  BRK_REQUIRE(p.B > 0 && p.N > 0 && p.Nk > 0 && p.N % p.Nk == 0 && p.S > 0 && p.M >= 1, BRK_E_ARG,
              "bad score shape B=%d N=%d Nk=%d S=%d M=%d", p.B, p.N, p.Nk, p.S, p.M);
  BRK_REQUIRE(p.R >= 1 && p.R <= 64 && (p.N / p.Nk) * p.R <= 256, BRK_E_ARG, "R=%d out of range", p.R);
  BRK_REQUIRE(p.D == 64 || p.D == 128, BRK_E_UNSUPPORTED, "head_dim %d not supported (64 or 128)", p.D);
  BRK_REQUIRE(p.dtype == BRK_BF16 || p.dtype == BRK_F32, BRK_E_UNSUPPORTED, "dtype %d", p.dtype);
  const int al = p.dtype == BRK_BF16 ? 8 : 4;
  BRK_REQUIRE(p.q.stride_s % al == 0 && p.q.stride_h % al == 0 && p.q.stride_b % al == 0 && p.k.stride_s % al == 0 &&
                  p.k.stride_h % al == 0 && p.k.stride_b % al == 0 && ((uintptr_t)p.q.ptr % 16 == 0) &&
                  ((uintptr_t)p.k.ptr % 16 == 0),
              BRK_E_ARG, "q/k rows must be 16-byte aligned");
  BRK_REQUIRE(p.B * p.Nk <= 65535, BRK_E_UNSUPPORTED, "B*Nk too large");
  return BRK_OK;
}

}  // namespace brk
