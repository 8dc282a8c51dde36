// BlockRank attention backward: workspace and choice of kernel, for training through the registered attention function.
// The reference gets these gradients from autograd over its eager / SDPA paths
// (src/blockrank/blockrank_std_attention.py:96-262, 472-650); the mathematics is that of the softmax
// attention backward restricted to each row's visible keys:
//
//   delta_i = dO_i . O_i            p_ij = exp(scale * q_i . k_j - lse_i)        dP_ij = dO_i . v_j
//   dS_ij = p_ij (dP_ij - delta_i)  dQ_i = scale * sum_j dS_ij k_j
//   dK_j = scale * sum_i dS_ij q_i  dV_j = sum_i p_ij dO_i     (i over the rows that see key j, all heads of the group)
//
// Visible keys of a row (the forward's pattern): block 0 is causal; a document block sees block 0 and
// itself causally; the last block sees every earlier block and itself causally.
//
//   bf16  attn_bwd_tc.cu (tcgen05) where a block fits its work item, else attn_bwd_mma.cu (warp-level MMA, blocks split
//         over CTAs)
//   fp32  attn_bwd_f32.cu (CUDA cores)
#include "brk_common.cuh"

namespace brk {

// scratch: delta [B, N, S]; bf16 only: fp32 dk, dv, of every slot ([B, Nk, S, D] each) for the warp-level kernels, of the prefix
// block ([B, Nk, max_block_len, D]) for the tcgen05 kernel of three blocks or more; fp32 dq of the last block's rows [B, N,
// max_block_len, D]; what the tcgen05 kernel needs beyond that
static size_t delta_bytes(const brk_attn_bwd_params& p) {
  return (((size_t)p.B * p.N * p.S * sizeof(float)) + 255) & ~(size_t)255;
}
static size_t acc_bytes(const brk_attn_bwd_params& p) { return (size_t)p.B * p.Nk * p.S * p.D * sizeof(float); }
static size_t dq_last_bytes(const brk_attn_bwd_params& p) { return (size_t)p.B * p.N * p.max_block_len * p.D * sizeof(float); }

static size_t sums_bytes(const brk_attn_bwd_params& p) {
  const bool prefix = attn_bwd_tc_supported(p) && p.M > 2;
  return 2 * (prefix ? (size_t)p.B * p.Nk * p.max_block_len * p.D * sizeof(float) : acc_bytes(p));
}

size_t attn_bwd_workspace(const brk_attn_bwd_params& p) {
  if (p.dtype == BRK_F32) return delta_bytes(p);
  return delta_bytes(p) + sums_bytes(p) + dq_last_bytes(p) + (attn_bwd_tc_supported(p) ? attn_bwd_tc_extra_bytes(p) : 0);
}

int attn_bwd_launch(const brk_attn_bwd_params& p, void* ws, size_t ws_bytes, int32_t* status, cudaStream_t st) {
  BRK_REQUIRE(ws != nullptr && ws_bytes >= attn_bwd_workspace(p) && ((uintptr_t)ws & 15) == 0, BRK_E_WORKSPACE,
              "workspace %zu < %zu bytes (or not 16-byte aligned)", ws_bytes, attn_bwd_workspace(p));
  unsigned char* const w = static_cast<unsigned char*>(ws);
  float* const delta = reinterpret_cast<float*>(w);
  if (p.dtype == BRK_F32) return attn_bwd_f32_launch(p, delta, st);
  float* const acc = reinterpret_cast<float*>(w + delta_bytes(p));
  unsigned char* const dq32 = w + delta_bytes(p) + sums_bytes(p);
  if (attn_bwd_tc_supported(p))
    return attn_bwd_tc_launch(p, delta, acc, reinterpret_cast<float*>(dq32), dq32 + dq_last_bytes(p), status, st);
  BRK_CUDA(cudaMemsetAsync(acc, 0, 2 * acc_bytes(p) + dq_last_bytes(p), st));
  return attn_bwd_mma_launch(p, delta, acc, acc + acc_bytes(p) / sizeof(float), reinterpret_cast<float*>(dq32), st);
}

}  // namespace brk
