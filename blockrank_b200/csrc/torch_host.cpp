// Native host path between PyTorch tensors and the C ABI (include/blockrank_b200.h).
//
// One call of the Python package is one call into this module: argument checks, output and scratch allocation
// (PyTorch's caching allocator, current stream), parameter structs, the C-ABI calls and -- for the registered
// attention function under autograd and for the early-exit ranker -- the sequence of such calls.  Written in Python the
// same steps cost 40-60 us per attention call, more than its kernels take on a short prompt.
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <ATen/cuda/tunable/Tunable.h>
#include <ATen/ops/addmm_cuda_dispatch.h>
#include <ATen/ops/mm_cuda_dispatch.h>
#include <c10/cuda/CUDAGuard.h>
#include <cublas_v2.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/extension.h>

#include <mutex>
#include <optional>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/blockrank_b200.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

// ---- errors -----------------------------------------------------------------------------------
// Raised as blockrank_b200's BlockRankLibraryError; argument errors are ValueErrors, CPU tensors RuntimeErrors.
struct LibError : std::runtime_error {
  using std::runtime_error::runtime_error;
};
PyObject *g_lib_error = nullptr, *g_oom_error = nullptr;  // BlockRankLibraryError, torch.OutOfMemoryError

#define BRK_VALUE(cond, ...)                                                  \
  do {                                                                        \
    if (!(cond)) C10_THROW_ERROR(ValueError, c10::str(__VA_ARGS__));          \
  } while (0)

const char* code_name(int rc) {
  switch (rc) {
    case -1: return "BRK_E_ARG";
    case -2: return "BRK_E_UNSUPPORTED";
    case -3: return "BRK_E_WORKSPACE";
    case -4: return "BRK_E_CUDA";
    case -5: return "BRK_E_DEVICE";
    case -6: return "BRK_E_TIMEOUT";
    default: return "error";
  }
}
void check(int rc, const char* what) {
  if (rc == 0) return;
  const std::string msg = c10::str(what, ": ", code_name(rc), ": ", brk_last_error());
  if (rc >= -3 && rc <= -1) C10_THROW_ERROR(ValueError, msg);
  throw LibError(msg);
}

void need_cuda(std::initializer_list<const Tensor*> ts) {
  for (const Tensor* t : ts)
    if (t != nullptr && t->defined())
      TORCH_CHECK(t->is_cuda(), "blockrank_b200 kernels run on CUDA tensors only (there is no CPU path)");
}
const Tensor* opt(const OptTensor& t) { return t.has_value() ? &*t : nullptr; }

// ---- parameter building -----------------------------------------------------------------------
int dtype_code(const Tensor& t) {
  if (t.scalar_type() == at::kBFloat16) return BRK_BF16;
  if (t.scalar_type() == at::kFloat) return BRK_F32;
  C10_THROW_ERROR(ValueError, c10::str("blockrank_b200 supports bfloat16 and float32, got ", t.scalar_type()));
}
void* stream_of(const Tensor& t) { return at::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

// starts and lengths of every block of B prompts: the kernels read B * M of each
void need_spans(const Tensor& start, const Tensor& length, int64_t B) {
  BRK_VALUE(start.scalar_type() == at::kInt && length.scalar_type() == at::kInt && start.sizes() == length.sizes() && start.dim() >= 1,
            "blk_start / blk_len must be int32 tensors of the same (B, M) shape");
  BRK_VALUE(start.numel() >= B * start.size(-1), "block spans of ", start.sizes(), " are too few for ", B, " prompts");
}

// (B, heads, S, D) tensor (any strides, innermost contiguous) -> brk_view
brk_view view_of(const Tensor& t) {
  BRK_VALUE(t.dim() == 4 && t.stride(3) == 1, "expected a (B, heads, S, D) tensor with contiguous head_dim");
  brk_view v;
  v.ptr = t.data_ptr();
  v.stride_b = t.stride(0);
  v.stride_h = t.stride(1);
  v.stride_s = t.stride(2);
  return v;
}
// (B, S, heads, D) tensor -> the same view
brk_view view_bshd(const Tensor& t) {
  BRK_VALUE(t.dim() == 4 && t.stride(3) == 1, "expected a (B, heads, S, D) tensor with contiguous head_dim");
  brk_view v;
  v.ptr = t.data_ptr();
  v.stride_b = t.stride(0);
  v.stride_h = t.stride(2);
  v.stride_s = t.stride(1);
  return v;
}
Tensor empty_bshd(const Tensor& like, int64_t B, int64_t S, int64_t heads, int64_t D) {
  return at::empty({B, S, heads, D}, like.options().requires_grad(false));
}
Tensor scratch(size_t bytes, const Tensor& like) {
  return at::empty({(int64_t)bytes}, like.options().dtype(at::kByte).requires_grad(false));
}

// One int32 status word per device, zeroed when created.  Every attention call passes it; the kernels set it (the first
// code written stays) when a bounded wait gives up or the block spans are malformed.
Tensor status_word(int device) {
  static std::mutex mu;
  static auto* words = new std::vector<Tensor>();  // (never destroyed: the CUDA context may be gone at exit)
  std::lock_guard<std::mutex> lock(mu);
  if ((int)words->size() <= device) words->resize(device + 1);
  Tensor& t = (*words)[device];
  if (!t.defined()) t = at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, device));
  return t;
}

std::tuple<Tensor, Tensor> spans_from_mask(const Tensor& mask) {
  need_cuda({&mask});
  BRK_VALUE(mask.dim() == 3, "block mask must be (B, M, H)");
  c10::cuda::CUDAGuard guard(mask.device());
  Tensor m8 = mask.scalar_type() == at::kBool ? mask.contiguous().view(at::kByte) : mask.ne(0).to(at::kByte).contiguous();
  const auto opts = m8.options().dtype(at::kInt);
  Tensor start = at::empty({m8.size(0), m8.size(1)}, opts), len = at::empty({m8.size(0), m8.size(1)}, opts);
  check(brk_spans_from_mask((const uint8_t*)m8.data_ptr(), (int)m8.size(0), (int)m8.size(1), (int)m8.size(2),
                            (int32_t*)start.data_ptr(), (int32_t*)len.data_ptr(), stream_of(m8)),
        "brk_spans_from_mask");
  return {start, len};
}

// ---- attention --------------------------------------------------------------------------------
std::tuple<Tensor, Tensor> attention(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& blk_start,
                                     const Tensor& blk_len, double scale, int64_t max_block_len, const OptTensor& out_in,
                                     bool return_lse, int64_t algo, int64_t max_query_len, const OptTensor& lse_in) {
  need_cuda({&q, &k, &v, &blk_start, &blk_len});
  BRK_VALUE(q.dim() == 4 && k.dim() == 4 && v.dim() == 4, "expected (B, heads, S, D) tensors");
  const int64_t B = q.size(0), N = q.size(1), S = q.size(2), D = q.size(3), Nk = k.size(1);
  BRK_VALUE(k.size(0) == B && k.size(2) == S && k.size(3) == D && v.sizes() == k.sizes(), "shape mismatch q", q.sizes(), " k",
            k.sizes(), " v", v.sizes());
  BRK_VALUE(k.scalar_type() == q.scalar_type() && v.scalar_type() == q.scalar_type(), "q, k, v must share a dtype");
  need_spans(blk_start, blk_len, B);
  c10::cuda::CUDAGuard guard(q.device());
  Tensor out = out_in.has_value() ? *out_in : empty_bshd(q, B, S, N, D);
  Tensor lse = lse_in.has_value() ? *lse_in
               : return_lse       ? at::empty({B, N, S}, q.options().dtype(at::kFloat).requires_grad(false))
                                  : Tensor();
  const Tensor bs = blk_start.contiguous(), bl = blk_len.contiguous();
  brk_attn_params p{};
  p.dtype = dtype_code(q);
  p.algo = (int32_t)algo;
  p.B = (int32_t)B; p.N = (int32_t)N; p.Nk = (int32_t)Nk; p.D = (int32_t)D; p.S = (int32_t)S;
  p.M = (int32_t)bs.size(-1);
  p.max_block_len = (int32_t)max_block_len;
  p.max_query_len = (int32_t)max_query_len;
  p.scale = (float)scale;
  p.q = view_of(q); p.k = view_of(k); p.v = view_of(v);
  p.o = view_bshd(out);
  p.lse = lse.defined() ? (float*)lse.data_ptr() : nullptr;
  p.blk_start = (const int32_t*)bs.data_ptr();
  p.blk_len = (const int32_t*)bl.data_ptr();
  p.status = (int32_t*)status_word(q.get_device()).data_ptr();
  const size_t nbytes = brk_attn_fwd_workspace_bytes(&p);
  Tensor ws = scratch(nbytes, q);
  check(brk_attn_fwd(&p, ws.data_ptr(), nbytes, stream_of(q)), "brk_attn_fwd");
  return {out, lse};
}

std::tuple<Tensor, Tensor, Tensor> attention_bwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& out,
                                                 const Tensor& d_out_in, const Tensor& lse_in, const Tensor& blk_start,
                                                 const Tensor& blk_len, double scale, int64_t max_block_len) {
  need_cuda({&q, &k, &v, &out, &d_out_in, &lse_in, &blk_start, &blk_len});
  BRK_VALUE(q.dim() == 4 && k.dim() == 4, "expected (B, heads, S, D) tensors");
  const int64_t B = q.size(0), N = q.size(1), S = q.size(2), D = q.size(3), Nk = k.size(1);
  BRK_VALUE(out.sizes() == at::IntArrayRef({B, S, N, D}) && d_out_in.sizes() == out.sizes(), "out / d_out must be (B,S,N,D) = ",
            at::IntArrayRef({B, S, N, D}), ", got ", out.sizes(), " / ", d_out_in.sizes());
  BRK_VALUE(lse_in.sizes() == at::IntArrayRef({B, N, S}) && lse_in.scalar_type() == at::kFloat,
            "lse must be the forward's fp32 (B, N, S) tensor");
  for (const Tensor* t : {&k, &v, &out, &d_out_in})
    BRK_VALUE(t->scalar_type() == q.scalar_type(), "q, k, v, out, d_out must share a dtype");
  need_spans(blk_start, blk_len, B);
  c10::cuda::CUDAGuard guard(q.device());
  const Tensor d_out = d_out_in.contiguous(), lse = lse_in.contiguous();  // (autograd may hand over expanded or transposed gradients)
  Tensor dq = empty_bshd(q, B, S, N, D).permute({0, 2, 1, 3});
  Tensor dk = empty_bshd(q, B, S, Nk, D).permute({0, 2, 1, 3});
  Tensor dv = empty_bshd(q, B, S, Nk, D).permute({0, 2, 1, 3});
  const Tensor bs = blk_start.contiguous(), bl = blk_len.contiguous();
  brk_attn_bwd_params p{};
  p.dtype = dtype_code(q);
  p.B = (int32_t)B; p.N = (int32_t)N; p.Nk = (int32_t)Nk; p.D = (int32_t)D; p.S = (int32_t)S;
  p.M = (int32_t)bs.size(-1);
  p.max_block_len = (int32_t)max_block_len;
  p.scale = (float)scale;
  p.q = view_of(q); p.k = view_of(k); p.v = view_of(v);
  p.o = view_bshd(out); p.d_o = view_bshd(d_out);
  p.lse = (const float*)lse.data_ptr();
  p.blk_start = (const int32_t*)bs.data_ptr();
  p.blk_len = (const int32_t*)bl.data_ptr();
  p.dq = view_of(dq); p.dk = view_of(dk); p.dv = view_of(dv);
  const size_t nbytes = brk_attn_bwd_workspace_bytes(&p);
  Tensor ws = scratch(nbytes, q);
  check(brk_attn_bwd_reporting(&p, ws.data_ptr(), nbytes, (int32_t*)status_word(q.get_device()).data_ptr(), stream_of(q)),
        "brk_attn_bwd");
  return {dq, dk, dv};
}

// ---- scores -----------------------------------------------------------------------------------
brk_score_params score_params(const Tensor& q, const Tensor& k, const Tensor& bs, const Tensor& bl, double scale, int64_t R,
                              double temperature) {
  need_spans(bs, bl, q.size(0));
  brk_score_params p{};
  p.dtype = dtype_code(q);
  p.B = (int32_t)q.size(0); p.N = (int32_t)q.size(1); p.Nk = (int32_t)k.size(1); p.D = (int32_t)q.size(3);
  p.S = (int32_t)q.size(2);
  p.M = (int32_t)bs.size(-1);
  p.R = (int32_t)R;
  p.scale = (float)scale;
  p.temperature = (float)temperature;
  p.q = view_of(q);
  p.k = view_of(k);
  p.blk_start = (const int32_t*)bs.data_ptr();
  p.blk_len = (const int32_t*)bl.data_ptr();
  return p;
}

std::tuple<Tensor, Tensor> doc_scores(const Tensor& q, const Tensor& k, const Tensor& blk_start, const Tensor& blk_len,
                                      const Tensor& rows_in, double scale, double temperature) {
  need_cuda({&q, &k, &blk_start, &blk_len, &rows_in});
  BRK_VALUE(rows_in.scalar_type() == at::kInt && rows_in.dim() == 2, "rows must be int32 (B, R)");
  BRK_VALUE(q.dim() == 4 && k.dim() == 4, "expected (B, heads, S, D) tensors");
  c10::cuda::CUDAGuard guard(q.device());
  const Tensor bs = blk_start.contiguous(), bl = blk_len.contiguous(), rows = rows_in.contiguous();
  brk_score_params p = score_params(q, k, bs, bl, scale, rows.size(1), temperature);
  p.S = (int32_t)q.size(2);
  const int64_t nd = p.M > 2 ? p.M - 2 : 0;
  const auto f32 = q.options().dtype(at::kFloat).requires_grad(false);
  Tensor mass = at::empty({q.size(0), q.size(1), rows.size(1), nd}, f32), logits = at::empty({q.size(0), nd}, f32);
  p.rows = (const int32_t*)rows.data_ptr();
  p.doc_mass = (float*)mass.data_ptr();
  p.logits = (float*)logits.data_ptr();
  const size_t nbytes = brk_doc_scores_workspace_bytes(&p);
  Tensor ws = scratch(nbytes > 8 ? nbytes : 8, q);
  check(brk_doc_scores(&p, ws.data_ptr(), nbytes, stream_of(q)), "brk_doc_scores");
  return {mass, logits};
}

// grid_h < 0: no grid (padding-free layout)
Tensor raw_scores(const Tensor& q, const Tensor& k, const Tensor& blk_start, const Tensor& blk_len, double scale,
                  int64_t num_last, int64_t grid_h) {
  need_cuda({&q, &k, &blk_start, &blk_len});
  BRK_VALUE(q.dim() == 4 && k.dim() == 4, "expected (B, heads, S, D) tensors");
  const int64_t B = q.size(0), N = q.size(1), S = q.size(2);
  const int64_t R = std::min(num_last, grid_h < 0 ? S : grid_h);
  c10::cuda::CUDAGuard guard(q.device());
  const Tensor bs = blk_start.contiguous(), bl = blk_len.contiguous();
  brk_score_params p = score_params(q, k, bs, bl, scale, R, 0.05);
  Tensor out = at::empty({B, N, R, S}, q.options().requires_grad(false));
  check(brk_raw_scores(&p, out.data_ptr(), stream_of(q)), "brk_raw_scores");
  return out;
}

std::tuple<Tensor, Tensor> raw_scores_bwd(const Tensor& q, const Tensor& k, const Tensor& d_raw_in, const Tensor& blk_start,
                                          const Tensor& blk_len, double scale, const OptTensor& dq_in, const OptTensor& dk_in) {
  need_cuda({&q, &k, &d_raw_in, opt(dq_in), opt(dk_in)});
  BRK_VALUE(q.dim() == 4 && k.dim() == 4 && d_raw_in.dim() == 4, "expected (B, heads, S, D) tensors");
  const int64_t B = q.size(0), N = q.size(1), S = q.size(2), D = q.size(3), Nk = k.size(1), R = d_raw_in.size(2);
  BRK_VALUE(d_raw_in.sizes() == at::IntArrayRef({B, N, R, S}) && d_raw_in.scalar_type() == q.scalar_type(), "d_raw must be (", B,
            ", ", N, ", R, ", S, ") ", q.scalar_type(), ", got ", d_raw_in.sizes(), " ", d_raw_in.scalar_type());
  const bool add = dq_in.has_value();
  BRK_VALUE(add == dk_in.has_value(), "give both dq and dk, or neither");
  c10::cuda::CUDAGuard guard(q.device());
  Tensor dq = add ? *dq_in : at::zeros({B, S, N, D}, q.options().requires_grad(false)).permute({0, 2, 1, 3});
  Tensor dk = add ? *dk_in : empty_bshd(q, B, S, Nk, D).permute({0, 2, 1, 3});
  const Tensor d_raw = d_raw_in.contiguous(), bs = blk_start.contiguous(), bl = blk_len.contiguous();
  brk_score_params p = score_params(q, k, bs, bl, scale, R, 0.05);
  const brk_view vq = view_of(dq), vk = view_of(dk);
  const size_t nbytes = brk_raw_scores_bwd_workspace_bytes(&p);
  Tensor ws = scratch(nbytes, q);
  check(brk_raw_scores_bwd(&p, d_raw.data_ptr(), &vq, &vk, add ? 1 : 0, ws.data_ptr(), nbytes, stream_of(q)),
        "brk_raw_scores_bwd");
  return {dq, dk};
}

// ---- autograd ---------------------------------------------------------------------------------
// An error of the library raised in a backward thread keeps its Python type.
[[noreturn]] void rethrow_as_python(const LibError& e) {
  pybind11::gil_scoped_acquire gil;
  PyErr_SetString(g_lib_error, e.what());
  python_error err;
  err.persist();
  throw err;
}

// Gradient of the raw logits in PyTorch operations, for a backward that is differentiated itself (create_graph).
std::tuple<Tensor, Tensor> raw_grad_graph(const Tensor& q, const Tensor& k, const Tensor& d_raw, double scale) {
  const int64_t B = q.size(0), N = q.size(1), S = q.size(2), D = q.size(3), Nk = k.size(1), R = d_raw.size(2);
  const Tensor g = (d_raw.to(at::kFloat) * scale).reshape({B, Nk, N / Nk, R, S});
  const Tensor q_last = q.narrow(2, S - R, R).to(at::kFloat).reshape({B, Nk, N / Nk, R, D});
  const Tensor dq = at::einsum("bkgrs,bksd->bkgrd", {g, k.to(at::kFloat)}).reshape({B, N, R, D}).to(q.scalar_type());
  return {at::constant_pad_nd(dq, {0, 0, S - R, 0}), at::einsum("bkgrs,bkgrd->bksd", {g, q_last}).to(k.scalar_type())};
}

// Backward of the attention output (brk_attn_bwd) and, where they were asked for, of the raw logits of the last R slots,
// (B,N,R,S) = scale * q[:, :, S-R:] k^T + a mask addend (std:219-233, 256-262): the addend is constant, so their gradient
// flows to q and k at every position (brk_raw_scores_bwd).  One node for both outputs: a pass that brings both gradients adds
// the second into the first instead of leaving two pairs of tensors for autograd to sum.  What an output saved is given back
// on its own, behind the pass that used it, so that the two can be differentiated in passes of their own.
struct AttentionNode : torch::autograd::Node {
  using List = torch::autograd::variable_list;
  using Saved = torch::autograd::SavedVariable;

  Saved q, k, v, out, lse, start, length;
  double scale = 0;
  int64_t max_block_len = 0;
  bool spent[2] = {false, true};  // output 0: attention, 1: raw logits (none: nothing saved for them)
  bool used[2] = {false, false};  // by the latest pass

  std::string name() const override { return "BlockRankAttentionBackward"; }

  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (int i = 0; i < 2; ++i) spent[i] |= used[i];
    if (spent[0])
      for (Saved* t : {&v, &out, &lse}) t->reset_data();
    if (spent[0] && spent[1])
      for (Saved* t : {&q, &k, &start, &length}) t->reset_data();
  }

  List apply(List&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    try {
      used[0] = grads[0].defined();
      used[1] = grads.size() > 1 && grads[1].defined();
      for (int i = 0; i < 2; ++i) TORCH_CHECK(!(used[i] && spent[i]), torch::autograd::ERR_BACKWARD_TWICE);
      Tensor dq, dk, dv;
      if (!used[0] && !used[1]) return {dq, dk, dv};
      const Tensor sq = q.unpack(), sk = k.unpack(), ss = start.unpack(), sl = length.unpack();
      const bool graph = at::GradMode::is_enabled();
      if (used[0]) {
        const Tensor so = out.unpack(shared_from_this()), sv = v.unpack(), slse = lse.unpack();
        at::NoGradGuard no_grad;
        std::tie(dq, dk, dv) = attention_bwd(sq, sk, sv, so, grads[0].to(so.scalar_type()), slse, ss, sl, scale, max_block_len);
      }
      if (used[1] && graph) {
        const auto [rq, rk] = raw_grad_graph(sq, sk, grads[1], scale);
        dq = used[0] ? dq + rq : rq;
        dk = used[0] ? dk + rk : rk;
      } else if (used[1]) {
        std::tie(dq, dk) = raw_scores_bwd(sq, sk, grads[1].to(sq.scalar_type()), ss, sl, scale,
                                          used[0] ? OptTensor(dq) : std::nullopt, used[0] ? OptTensor(dk) : std::nullopt);
      }
      return {dq, dk, dv};
    } catch (const LibError& e) {
      rethrow_as_python(e);
    }
  }
};

// num_last < 0: no raw logits.  spans: int32 (2, B, M) [starts; lengths], (2, M) for one prompt.  Returns (out, raw or None).
std::tuple<Tensor, OptTensor> attention_forward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& spans,
                                                double scale, int64_t max_block_len, int64_t max_query_len, int64_t algo,
                                                int64_t num_last, int64_t grid_h) {
  BRK_VALUE(spans.dim() >= 2 && spans.size(0) >= 2, "block spans must be an int32 (2, B, M) tensor, or (2, M) for one prompt");
  const Tensor start = spans.select(0, 0), length = spans.select(0, 1);
  const bool train = torch::autograd::compute_requires_grad(q, k, v);
  if (train)
    for (const Tensor* t : {&q, &k, &v})
      TORCH_CHECK_NOT_IMPLEMENTED(!t->_fw_grad(/*level=*/0).defined(), "BlockRank attention has no forward-mode derivative");
  Tensor out, lse, raw;
  {
    at::AutoGradMode no_grad(false);
    std::tie(out, lse) = attention(q, k, v, start, length, scale, max_block_len, std::nullopt, train, algo, max_query_len, std::nullopt);
    if (num_last >= 0) raw = raw_scores(q, k, start, length, scale, num_last, grid_h);
  }
  if (train) {
    std::shared_ptr<AttentionNode> node(new AttentionNode(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(q, k, v));
    node->q = AttentionNode::Saved(q, false);
    node->k = AttentionNode::Saved(k, false);
    node->v = AttentionNode::Saved(v, false);
    node->lse = AttentionNode::Saved(lse, false);
    node->start = AttentionNode::Saved(start, false);
    node->length = AttentionNode::Saved(length, false);
    node->scale = scale;
    node->max_block_len = max_block_len;
    torch::autograd::set_history(out, node);
    if (raw.defined()) {
      node->spent[1] = false;
      torch::autograd::set_history(raw, node);
    }
    node->out = AttentionNode::Saved(out, true);
  }
  return {out, raw.defined() ? OptTensor(raw) : std::nullopt};
}

// ---- runner helpers ---------------------------------------------------------------------------
Tensor rmsnorm(const Tensor& x, const Tensor& weight, double eps, const OptTensor& residual, const OptTensor& out_in) {
  need_cuda({&x, &weight, opt(residual)});
  BRK_VALUE(x.is_contiguous() && (!residual.has_value() || residual->is_contiguous()), "rmsnorm expects contiguous rows");
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t hidden = x.size(-1), rows = hidden > 0 ? x.numel() / hidden : 0;
  Tensor out = out_in.has_value() ? *out_in : at::empty_like(x);
  check(brk_rmsnorm(dtype_code(x), x.data_ptr(), residual.has_value() ? residual->data_ptr() : nullptr, weight.data_ptr(),
                    out.data_ptr(), rows, (int32_t)hidden, (float)eps, stream_of(x)),
        "brk_rmsnorm");
  return out;
}

void rope_(const OptTensor& q, const OptTensor& k, const Tensor& pos, const Tensor& inv_freq) {
  if (!q.has_value() && !k.has_value()) return;
  const Tensor& ref = q.has_value() ? *q : *k;
  need_cuda({&ref, &pos, &inv_freq});
  BRK_VALUE(ref.dim() == 3, "rope_ expects (T, heads, D) views with contiguous heads");
  const int64_t T = ref.size(0), D = ref.size(2);
  for (const Tensor* t : {opt(q), opt(k)})
    if (t != nullptr)
      BRK_VALUE(t->dim() == 3 && t->size(0) == T && t->size(2) == D && t->stride(2) == 1 && t->stride(1) == D,
                "rope_ expects (T, heads, D) views with contiguous heads");
  BRK_VALUE(pos.scalar_type() == at::kInt && inv_freq.scalar_type() == at::kFloat && pos.numel() == T && pos.is_contiguous(),
            "pos must be contiguous int32 (T,) and inv_freq float32");
  c10::cuda::CUDAGuard guard(ref.device());
  check(brk_rope(dtype_code(ref), q.has_value() ? q->data_ptr() : nullptr, q.has_value() ? q->stride(0) : 0,
                 q.has_value() ? (int32_t)q->size(1) : 0, k.has_value() ? k->data_ptr() : nullptr,
                 k.has_value() ? k->stride(0) : 0, k.has_value() ? (int32_t)k->size(1) : 0, (int32_t)D,
                 (const int32_t*)pos.data_ptr(), (const float*)inv_freq.data_ptr(), T, stream_of(ref)),
        "brk_rope");
}

Tensor silu_mul(const Tensor& gate_up, const OptTensor& out_in) {
  need_cuda({&gate_up});
  BRK_VALUE(gate_up.is_contiguous(), "silu_mul expects a contiguous (rows, 2*I) tensor");
  c10::cuda::CUDAGuard guard(gate_up.device());
  const int64_t inter = gate_up.size(-1) / 2, rows = inter > 0 ? gate_up.numel() / (2 * inter) : 0;
  Tensor out;
  if (out_in.has_value()) {
    out = *out_in;
  } else {
    auto shape = gate_up.sizes().vec();
    shape.back() = inter;
    out = at::empty(shape, gate_up.options());
  }
  check(brk_silu_mul(dtype_code(gate_up), gate_up.data_ptr(), out.data_ptr(), rows, (int32_t)inter, stream_of(gate_up)),
        "brk_silu_mul");
  return out;
}

// ---- early-exit ranker --------------------------------------------------------------------------
// PyTorch's GEMMs with the autograd layers of its dispatcher left out: nothing here is ever differentiated.
struct NoAutograd {
  at::NoGradGuard no_grad;
  at::AutoDispatchBelowADInplaceOrView below_autograd;
};


// Are PyTorch's switches for bf16 products where they start out?  The call below knows none of them.
bool default_products() {
  auto& ctx = at::globalContext();
  const auto blas = ctx.blasPreferredBackend();
  return ctx.allowBF16ReductionCuBLAS() == at::CuBLASReductionOption::AllowReducedPrecisionWithSplitK &&
         (blas == at::BlasBackend::Default || blas == at::BlasBackend::Cublas) && !ctx.deterministicAlgorithms() &&
         !at::cuda::tunable::getTuningContext()->IsTunableOpEnabled();
}

// out (+)= x w^T for row-major x (T, K), w (n, K) on the current device: for bf16, and while nobody has set a switch, cuBLAS on
// PyTorch's handle (its stream and workspace), the call that torch.mm / addmm end in without their host path.
void gemm_nt(Tensor& out, const Tensor& x, const Tensor& w, bool add) {
  const int64_t T = x.size(0), K = x.size(1), n = w.size(0);
  const bool plain = out.is_contiguous() && x.is_contiguous() && w.is_contiguous() && w.dim() == 2 && w.size(1) == K &&
                     out.scalar_type() == at::kBFloat16 && x.scalar_type() == at::kBFloat16 && w.scalar_type() == at::kBFloat16 &&
                     T > 0 && K > 0 && n > 0 && std::max({T, K, n}) < (1ll << 31) && default_products();
  if (!plain) {
    if (add) at::cuda::addmm_(out, x, w.t(), 1, 1);
    else at::cuda::mm_out(out, x, w.t());
    return;
  }
  const float one = 1.f, beta = add ? 1.f : 0.f;
  const cublasStatus_t rc = cublasGemmEx(at::cuda::getCurrentCUDABlasHandle(), CUBLAS_OP_T, CUBLAS_OP_N, (int)n, (int)T, (int)K, &one,
                                         w.data_ptr(), CUDA_R_16BF, (int)K, x.data_ptr(), CUDA_R_16BF, (int)K, &beta, out.data_ptr(),
                                         CUDA_R_16BF, (int)n, CUBLAS_COMPUTE_32F, CUBLAS_GEMM_DEFAULT_TENSOR_OP);
  TORCH_CHECK(rc == CUBLAS_STATUS_SUCCESS, "cublasGemmEx failed (", (int)rc, ")");
}
Tensor mm_nt(const Tensor& x, const Tensor& w) {
  Tensor out = at::empty({x.size(0), w.size(0)}, x.options());
  gemm_nt(out, x, w, false);
  return out;
}

// input norm, fused QKV projection, RoPE on q and k in place: (T, (N + 2 Nk) D)
Tensor layer_qkv(const Tensor& h, const Tensor& ln1, const Tensor& wqkv, const Tensor& pos, const Tensor& inv_freq, int64_t N,
                 int64_t Nk, int64_t D, double eps) {
  NoAutograd guard;
  c10::cuda::CUDAGuard device(h.device());
  Tensor qkv = mm_nt(rmsnorm(h, ln1, eps, std::nullopt, std::nullopt), wqkv);
  const int64_t T = qkv.size(0), row = qkv.stride(0), at0 = qkv.storage_offset();
  rope_(qkv.as_strided({T, N, D}, {row, D, 1}, at0), qkv.as_strided({T, Nk, D}, {row, D, 1}, at0 + N * D), pos, inv_freq);
  return qkv;
}

Tensor layer_attention(const Tensor& qkv, const Tensor& blk_start, const Tensor& blk_len, int64_t B, int64_t S, int64_t N,
                       int64_t Nk, int64_t D, int64_t max_block_len, int64_t max_query_len, int64_t algo) {
  NoAutograd guard;
  const int64_t row = qkv.stride(0), at0 = qkv.storage_offset();
  auto heads = [&](int64_t n, int64_t first) {
    return qkv.as_strided({B, n, S, D}, {S * row, D, row, 1}, at0 + first * D);
  };
  return std::get<0>(attention(heads(N, 0), heads(Nk, N), heads(Nk, N + Nk), blk_start, blk_len, 1.0 / std::sqrt((double)D),
                               max_block_len, std::nullopt, false, algo, max_query_len, std::nullopt));
}

// h += o_proj(attn); h += down_proj(silu(gate) * up) of its norm.  Both residual additions happen in the epilogue of the
// GEMM that produces the branch (C = C + A B, added in fp32 before the rounding).
void layer_rest(Tensor& h, const Tensor& attn, const Tensor& wo, const Tensor& ln2, const Tensor& wgu, const Tensor& wd,
                double eps) {
  NoAutograd guard;
  c10::cuda::CUDAGuard device(h.device());
  gemm_nt(h, attn.view({h.size(0), wo.size(1)}), wo, true);
  const Tensor x = rmsnorm(h, ln2, eps, std::nullopt, std::nullopt);
  gemm_nt(h, silu_mul(mm_nt(x, wgu), std::nullopt), wd, true);
}

// layers: {ln1, wqkv, wo, ln2, wgu, wd} of every layer in front of the scoring layer.  ids (B, S), pos int32 (B S,).
Tensor hidden_states(const Tensor& embed, const Tensor& ids, const std::vector<std::vector<Tensor>>& layers, const Tensor& pos,
                     const Tensor& inv_freq, const Tensor& blk_start, const Tensor& blk_len, int64_t max_block_len,
                     int64_t max_query_len, int64_t N, int64_t Nk, int64_t D, double eps, int64_t algo) {
  NoAutograd guard;
  c10::cuda::CUDAGuard device(embed.device());
  const int64_t B = ids.size(0), S = ids.size(1);
  Tensor h = at::embedding(embed, ids.reshape({B * S}));
  for (const auto& L : layers) {
    const Tensor attn = layer_attention(layer_qkv(h, L.at(0), L.at(1), pos, inv_freq, N, Nk, D, eps), blk_start, blk_len, B, S,
                                        N, Nk, D, max_block_len, max_query_len, algo);
    layer_rest(h, attn, L.at(2), L.at(3), L.at(4), L.at(5), eps);
  }
  return h;
}

// The scoring layer up to the score epilogue: keys of every token, queries of the signal rows, both rotated; and the
// index of each query row inside q.  pos (B, S); signal_rows (B, R), or (1, R): the same rows of every prompt.
// Returns (q (B,N,R,D), k (B,Nk,S,D), rows int32 (B,R)).
std::tuple<Tensor, Tensor, Tensor> score_qk(const Tensor& h, const Tensor& pos, const Tensor& signal_rows, const Tensor& ln1,
                                            const Tensor& wq, const Tensor& wk, const Tensor& inv_freq, int64_t N, int64_t Nk,
                                            int64_t D, double eps) {
  NoAutograd guard;
  c10::cuda::CUDAGuard device(h.device());
  need_cuda({&h, &pos, &signal_rows});
  BRK_VALUE(signal_rows.scalar_type() == at::kInt && signal_rows.dim() == 2 && pos.scalar_type() == at::kInt && pos.is_contiguous(),
            "signal_rows must be int32 (B, R) and positions contiguous int32");
  BRK_VALUE(pos.dim() == 2 && h.dim() == 2 && h.size(0) == pos.numel(), "positions must be (B, S) for hidden states (B S, hidden), got ",
            pos.sizes(), " and ", h.sizes());
  const int64_t B = pos.size(0), R = signal_rows.size(1), T = h.size(0), S = pos.size(1);
  BRK_VALUE(signal_rows.size(0) == B || signal_rows.size(0) == 1, "signal_rows must be (B, R) or (1, R), got ", signal_rows.sizes(),
            " for ", B, " prompts");
  const Tensor x = rmsnorm(h, ln1, eps, std::nullopt, std::nullopt), rows = signal_rows.expand({B, R}).contiguous();
  Tensor k = mm_nt(x, wk);
  Tensor xs = at::empty({B * R, x.size(1)}, x.options()), ps = at::empty({B * R}, pos.options()), local = at::empty({B, R}, pos.options());
  check(brk_signal_rows(dtype_code(x), x.data_ptr(), (int32_t)x.size(1), (const int32_t*)pos.data_ptr(),
                        (const int32_t*)rows.data_ptr(), (int32_t)B, (int32_t)S, (int32_t)R, xs.data_ptr(),
                        (int32_t*)ps.data_ptr(), (int32_t*)local.data_ptr(), (int32_t*)status_word(x.get_device()).data_ptr(),
                        stream_of(x)),
        "brk_signal_rows");
  Tensor q = mm_nt(xs, wq);
  rope_(q.view({B * R, N, D}), std::nullopt, ps, inv_freq);
  rope_(std::nullopt, k.view({T, Nk, D}), pos, inv_freq);  // (pos: T of them, contiguous)
  return {q.view({B, R, N, D}).permute({0, 2, 1, 3}), k.view({B, S, Nk, D}).permute({0, 2, 1, 3}), local};
}

// Host tensors of a batch -> device: (ids, positions int32, start, length, signal rows), and the longest query block.
// They travel in one copy out of a pinned buffer (five copies and a conversion kernel were 40 us of a short request).
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, int64_t> upload(const Tensor& ids, const Tensor& pos, const Tensor& spans,
                                                                   const Tensor& rows, const c10::Device& device) {
  NoAutograd guard;
  BRK_VALUE(spans.dim() == 3 && spans.size(0) == 2 && spans.scalar_type() == at::kInt, "block_spans must be int32 (2, B, M)");
  const int64_t B = spans.size(1), M = spans.size(2);
  bool packable = ids.scalar_type() == at::kLong && rows.scalar_type() == at::kInt &&
                  (pos.scalar_type() == at::kLong || pos.scalar_type() == at::kInt);
  for (const Tensor* t : {&ids, &pos, &spans, &rows}) packable = packable && t->is_cpu() && t->is_contiguous();
  if (!packable) {
    const Tensor d_ids = ids.to(device, ids.scalar_type(), true), d_pos = pos.to(device, pos.scalar_type(), true).to(at::kInt);
    const Tensor d_spans = spans.to(device, spans.scalar_type(), true), d_rows = rows.to(device, at::kInt, true);
    return {d_ids, d_pos, d_spans.select(0, 0), d_spans.select(0, 1), d_rows, spans.select(0, 1).select(1, M - 1).max().item().toLong()};
  }
  const int64_t n_ids = ids.numel(), n_pos = pos.numel(), n_spans = spans.numel(), n_rows = rows.numel();
  Tensor stage = at::empty({8 * n_ids + 4 * (n_pos + n_spans + n_rows)}, at::TensorOptions().dtype(at::kByte).pinned_memory(true));
  char* w = static_cast<char*>(stage.data_ptr());
  memcpy(w, ids.data_ptr(), 8 * n_ids);
  int32_t* p = reinterpret_cast<int32_t*>(w + 8 * n_ids);
  if (pos.scalar_type() == at::kLong) {
    const int64_t* src = static_cast<const int64_t*>(pos.data_ptr());
    for (int64_t i = 0; i < n_pos; ++i) p[i] = (int32_t)src[i];
  } else {
    memcpy(p, pos.data_ptr(), 4 * n_pos);
  }
  memcpy(p + n_pos, spans.data_ptr(), 4 * n_spans);
  memcpy(p + n_pos + n_spans, rows.data_ptr(), 4 * n_rows);
  const Tensor d = stage.to(device, at::kByte, /*non_blocking=*/true);
  const Tensor d32 = d.narrow(0, 8 * n_ids, 4 * (n_pos + n_spans + n_rows)).view(at::kInt);
  auto part = [&](int64_t first, at::IntArrayRef sizes) {
    int64_t n = 1;
    for (int64_t x : sizes) n *= x;
    return d32.narrow(0, first, n).view(sizes);
  };
  const int32_t* len = static_cast<const int32_t*>(spans.data_ptr()) + B * M;
  int64_t longest = 0;
  for (int64_t b = 0; b < B; ++b) longest = std::max<int64_t>(longest, len[b * M + M - 1]);
  return {d.narrow(0, 0, 8 * n_ids).view(at::kLong).view(ids.sizes()), part(0, pos.sizes()), part(n_pos, {B, M}),
          part(n_pos + B * M, {B, M}), part(n_pos + n_spans, rows.sizes()), longest};
}

// Scores and the indices of the k best documents -> host, with one copy and one synchronisation, after which a problem a
// kernel reported is raised.
std::tuple<Tensor, Tensor> download(const Tensor& logits_in, int64_t k_in) {
  NoAutograd guard;
  c10::cuda::CUDAGuard device(logits_in.device());
  const Tensor logits = logits_in.contiguous();
  const int64_t B = logits.size(0), nd = logits.size(1), k = std::min(k_in, nd);
  const Tensor word = status_word(logits.get_device());
  const auto stream = at::cuda::getCurrentCUDAStream(logits.get_device());
  const size_t nl = logits.nbytes(), at_top = (nl + 15) & ~(size_t)15, nt = (size_t)B * k * 8, at_word = at_top + ((nt + 15) & ~(size_t)15);
  const auto bytes = at::TensorOptions().dtype(at::kByte);
  Tensor stage = at::empty({(int64_t)(at_word + 16)}, bytes.pinned_memory(true));
  char* const base = static_cast<char*>(stage.data_ptr());
  Tensor dev;  // alive until the copy is complete
  if (B > 0 && k > 0 && nd <= BRK_RANK_PACK_DOCS) {
    dev = at::empty({(int64_t)(at_word + 16)}, bytes.device(logits.device()));
    char* const d = static_cast<char*>(dev.data_ptr());
    check(brk_rank_pack((const float*)logits.data_ptr(), (int32_t)B, (int32_t)nd, (int32_t)k, (float*)d, (int64_t*)(d + at_top),
                        (const int32_t*)word.data_ptr(), (int32_t*)(d + at_word), stream.stream()),
          "brk_rank_pack");
    C10_CUDA_CHECK(cudaMemcpyAsync(base, d, at_word + 4, cudaMemcpyDeviceToHost, stream));
  } else {
    dev = std::get<1>(at::topk(logits, k, -1));
    C10_CUDA_CHECK(cudaMemcpyAsync(base, logits.data_ptr(), nl, cudaMemcpyDeviceToHost, stream));
    C10_CUDA_CHECK(cudaMemcpyAsync(base + at_top, dev.data_ptr(), nt, cudaMemcpyDeviceToHost, stream));
    C10_CUDA_CHECK(cudaMemcpyAsync(base + at_word, word.data_ptr(), 4, cudaMemcpyDeviceToHost, stream));
  }
  C10_CUDA_CHECK(cudaStreamSynchronize(stream));
  Tensor h_logits = at::empty(logits.sizes(), logits.options().device(at::kCPU));
  Tensor h_top = at::empty({B, k}, at::TensorOptions().dtype(at::kLong));
  memcpy(h_logits.data_ptr(), base, nl);
  memcpy(h_top.data_ptr(), base + at_top, nt);
  int32_t code;
  memcpy(&code, base + at_word, 4);
  if (code != 0) check(brk_status_poll((int32_t*)word.data_ptr(), stream.stream()), "brk_status_poll");
  return {h_logits, h_top};
}

// A ranking request from host tensors to host results: what MistralPrefillRanker.rank_host does, in one call.
// score_layer: {ln1, wq, wk} of the scoring layer.
std::tuple<Tensor, Tensor> rank(const Tensor& embed, const std::vector<std::vector<Tensor>>& layers,
                                const std::vector<Tensor>& score_layer, const Tensor& inv_freq, const Tensor& ids, const Tensor& pos,
                                const Tensor& spans, const Tensor& rows, int64_t max_block_len, int64_t N, int64_t Nk, int64_t D,
                                double eps, int64_t algo, double temperature, int64_t k) {
  c10::cuda::CUDAGuard device(embed.device());
  const auto [d_ids, d_pos, start, len, d_rows, longest] = upload(ids, pos, spans, rows, embed.device());
  BRK_VALUE(d_ids.dim() == 2 && d_pos.sizes() == d_ids.sizes(), "input_ids and position_ids must be (B, S), got ", d_ids.sizes(), " and ",
            d_pos.sizes());
  const Tensor h = hidden_states(embed, d_ids, layers, d_pos.reshape({-1}), inv_freq, start, len, max_block_len, longest, N, Nk, D, eps, algo);
  const auto [q, kk, local] = score_qk(h, d_pos.contiguous(), d_rows, score_layer.at(0), score_layer.at(1), score_layer.at(2), inv_freq, N, Nk, D, eps);
  return download(std::get<1>(doc_scores(q, kk, start, len, local, 1.0 / std::sqrt((double)D), temperature)), k);
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  namespace py = pybind11;
  py::register_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (const LibError& e) {
      PyErr_SetString(g_lib_error, e.what());
    } catch (const c10::OutOfMemoryError& e) {
      PyErr_SetString(g_oom_error, e.what_without_backtrace());
    } catch (const c10::ValueError& e) {
      PyErr_SetString(PyExc_ValueError, e.what_without_backtrace());
    } catch (const c10::NotImplementedError& e) {
      PyErr_SetString(PyExc_NotImplementedError, e.what_without_backtrace());
    } catch (const c10::IndexError& e) {
      PyErr_SetString(PyExc_IndexError, e.what_without_backtrace());
    } catch (const c10::Error& e) {
      PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
    }
  });
  m.def("set_error_classes", [](py::object lib, py::object oom) {
    g_lib_error = lib.release().ptr();
    g_oom_error = oom.release().ptr();
  });
  m.def("launch_count", &brk_launch_count);
  // Other Python threads run meanwhile: a launch blocks once the device's queue is full, and a ranking request waits for its
  // results.
  auto def = [&m](const char* name, auto f) { m.def(name, f, py::call_guard<py::gil_scoped_release>()); };
  def("status_word", &status_word);
  def("spans_from_mask", &spans_from_mask);
  def("attention", &attention);
  def("attention_bwd", &attention_bwd);
  def("attention_forward", &attention_forward);
  def("doc_scores", &doc_scores);
  def("raw_scores", &raw_scores);
  def("raw_scores_bwd", &raw_scores_bwd);
  def("rmsnorm", &rmsnorm);
  def("rope_", &rope_);
  def("silu_mul", &silu_mul);
  def("layer_qkv", &layer_qkv);
  def("layer_attention", &layer_attention);
  def("layer_rest", &layer_rest);
  def("hidden_states", &hidden_states);
  def("score_qk", &score_qk);
  def("upload", &upload);
  def("download", &download);
  def("rank", &rank);
}
