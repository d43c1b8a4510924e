// Shared declarations of the native op layer: the autograd nodes of the public ops, written against the
// C++ tensor API and launching the kernels of liberi_b200_kernels.so through their C entry points.
//
// What bounds it: a training step at a few hundred tokens is a chain of launches of 3-20 us each, and the
// same nodes written in Python (an autograd.Function, a ctypes call with one setattr per argument) took
// 20-30 us of host time per launch. Inside a node a launch costs 2-4 us here and the backward runs without the
// interpreter lock; the Python of a model between its nodes is not in that figure (a whole training pass of a small
// model comes to 12 us per launch).
#pragma once
#include <torch/extension.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/forward_grad.h>

#include <atomic>
#include <optional>
#include <tuple>
#include <vector>

#include "../attn_args.h"
#include "../gemm_args.h"

namespace eri_ops {

using at::Tensor;
using OptT = std::optional<Tensor>;
using torch::autograd::AutogradContext;
using torch::autograd::Variable;
using torch::autograd::variable_list;

// Kernel entry points, resolved from the library Python loaded (release or bounds-checked build).
#define ERI_FUNCS(X)                                                                                              \
  X(eri_norm_modulate_fwd, (const void*, const void*, const void*, const void*, const void*, void*, float*,      \
                            float*, int, int, int, int, float, int, void*))                                      \
  X(eri_norm_modulate_bwd, (const void*, const void*, const void*, const void*, const void*, const float*,       \
                            const float*, void*, float*, float*, float*, float*, int, int, int, int, int, void*)) \
  X(eri_norm_modulate_fwd_warp, (const void*, const void*, const void*, const void*, const void*, void*, float*, \
                                 float*, int, int, int, int, float, int, void*))                                 \
  X(eri_norm_modulate_bwd_warp_add, (const void*, const void*, const void*, const void*, const float*,           \
                                     const float*, void*, const void*, int, int, int, int, int, void*))          \
  X(eri_qknorm_rope_fwd, (const void*, const void*, const void*, const float*, const float*, void*, void*,       \
                          void*, int, int, int, int, int, int, float, int, int, void*))                          \
  X(eri_qknorm_rope_bwd, (const void*, const void*, const void*, const void*, const void*, const void*,          \
                          const float*, const float*, void*, float*, float*, int, int, int, int, int, int,       \
                          float, int, int, int, void*))                                                          \
  X(eri_gate_residual, (const void*, const void*, const void*, void*, long long, int, int, int, void*))          \
  X(eri_act_fwd, (const void*, void*, long long, int, void*))                                                    \
  X(eri_act_bwd, (const void*, const void*, void*, long long, int, void*))                                       \
  X(eri_act_fwd_rows, (const void*, long long, void*, long long, int, int, int, void*))                          \
  X(eri_act_bwd_rows, (const void*, long long, const void*, long long, void*, long long, int, int, int, void*))  \
  X(eri_glu_fwd, (const void*, void*, int, int, int, int, void*))                                                \
  X(eri_glu_bwd, (const void*, const void*, void*, int, int, int, int, void*))                                   \
  X(eri_mse_fwd_bwd, (const void*, const void*, const float*, float*, void*, long long, long long, float, void*)) \
  X(eri_gn_fwd, (const void*, const void*, const void*, const void*, const void*, void*, float*, float*, float*, \
                 int, int, int, int, float, int, void*))                                                         \
  X(eri_gn_bwd, (const void*, const void*, const void*, const void*, const void*, const void*, const float*,     \
                 const float*, void*, void*, void*, void*, void*, float*, int, int, int, int, int, int, void*))  \
  X(eri_add_bias, (const void*, const void*, const void*, const void*, void*, long long, int, void*))            \
  X(eri_conv_weight_order, (const void*, void*, int, int, int, int, void*))                                      \
  X(eri_upsample2x, (const void*, void*, long long, int, int, int, void*))                                       \
  X(eri_gemm_skinny, (const void*, long long, const void*, long long, void*, int, int, int, int, float, void*))  \
  X(eri_gemm_rank_stream, (const void*, long long, const void*, long long, void*, int, int, int, int, float,     \
                           void*))                                                                               \
  X(eri_gemm_rank_stream2, (const void*, long long, const void*, long long, void*, int, int, float, const void*, \
                            long long, const void*, long long, void*, int, int, float, int, int, void*))         \
  X(eri_gemm_tokred, (const void*, long long, const void*, long long, void*, int, int, int, int, float, int,     \
                      int, long long, void*))                                                                    \
  X(eri_gemm_bf16, (const EriGemmArgs*, void*))                                                                  \
  X(eri_gemm_few_bf16, (const EriGemmArgs*, void*))                                                              \
  X(eri_gemm2_bf16, (const EriGemmArgs*, void*))                                                                 \
  X(eri_gemm2_bf16_group2, (const EriGemmArgs*, const EriGemmArgs*, void*))                                      \
  X(eri_batched_transpose, (const void*, int, int, void*))                                                       \
  X(eri_col_sum, (const void*, long long, void*, int, int, int, void*))                                          \
  X(eri_col_norm_grad, (const void*, const void*, const float*, const float*, void*, void*, int, int, int, int,  \
                        void*))                                                                                  \
  X(eri_col_dot, (const void*, const void*, void*, int, int, int, void*))                                        \
  X(eri_flash_attn_fwd_pair, (const void*, const void*, const void*, void*, float*, int, int, int, int, int,     \
                              float, int, void*))                                                                \
  X(eri_rows_wgrad, (const void*, int, const void*, int, void*, int, int, int, int, int, float, void*))          \
  X(eri_rows_dgrad, (const void*, int, const void*, int, float*, int, int, int, int, void*))                     \
  X(eri_gemv_bf16, (const void*, const void*, const void*, void*, int, int, int, int, int, int, int, int, void*)) \
  X(eri_flash_attn_bias_fwd, (const void*, const void*, const void*, void*, const void*, long long, long long,   \
                              long long, int, int, int, int, int, int, float, const EriAttnStrides*, void*))     \
  X(eri_flash_attn_wide_fwd, (const void*, const void*, const void*, void*, int, int, int, int, float,           \
                              const EriAttnStrides*, void*))                                                     \
  X(eri_norm_rope_fwd, (const void*, const void*, long long, const void*, const void*, const float*, const float*, \
                        long long, void*, void*, float*, int, int, int, float, void*))                           \
  X(eri_norm_rope_bwd, (const void*, const void*, long long, const void*, const void*, const float*, const float*, \
                        long long, const float*, const void*, const void*, void*, void*, long long, int, int, int, \
                        void*))                                                                                  \
  X(eri_flash_attn_fwd_strided, (const void*, const void*, const void*, void*, float*, const float*, int, int,   \
                                 int, int, int, float, const EriAttnStrides*, void*))                            \
  X(eri_flash_attn_bwd_strided, (const void*, const void*, const void*, const void*, const void*, const float*,  \
                                 float*, float*, void*, void*, void*, const float*, int, int, int, int, int,     \
                                 float, const EriAttnStrides*, void*))

struct Lib {
  long long (*eri_gn_workspace)(int, int, int, int, int) = nullptr;
#define ERI_DECL(name, args) int(*name) args = nullptr;
  ERI_FUNCS(ERI_DECL)
#undef ERI_DECL
};
extern Lib L;
extern std::atomic<long long> g_launches;

// Switches and rules of ops/functional.py that the nodes honour, evaluated there at every call. From kFewTilesShift up: the
// most 256 x 256 tiles that a product may have and still run on the one-CTA kernel.
enum Flag : int { kPdl = 1, kRankStream = 2, kPair = 4, kGroup = 8, kActOutside = 16, kWgrad = 32, kAccumGrad = 64,
                  kNativeGemm = 128 };
constexpr int kFewTilesShift = 8;

inline void check(int code, const char* what) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  TORCH_CHECK(code == 0, what, " failed with code ", code);
}
inline void* stream() { return (void*)c10::cuda::getCurrentCUDAStream().stream(); }
inline const void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
inline void* mptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
inline Tensor opt(const OptT& t) { return t.has_value() ? *t : Tensor(); }
inline Tensor contig(const Tensor& t) { return !t.defined() || t.is_contiguous() ? t : t.contiguous(); }
inline bool al16(const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0; }
// contiguous and on a 16-byte boundary (a contiguous slice may start anywhere)
inline Tensor contig16(const Tensor& t) {
  if (!t.defined()) return t;
  Tensor c = contig(t);
  return al16(c) ? c : c.clone();
}
// bytes from t's first element to the end of its storage (what a kernel may touch through its pointer)
inline long long extent(const Tensor& t) {
  return t.defined() ? (long long)t.storage().nbytes() - t.storage_offset() * (long long)t.element_size() : 0;
}
inline bool bf16_cuda(const Tensor& t) { return !t.defined() || (t.is_cuda() && t.scalar_type() == at::kBFloat16); }
// a [M, K] operand the tensor-core kernels can read in place
inline bool rows_ok(const Tensor& t) {
  return t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.dim() == 2 && t.stride(1) == 1 && t.stride(0) % 8 == 0 &&
         al16(t);
}
inline Tensor empty_bf16(at::IntArrayRef s, const Tensor& like) {
  return at::empty(s, like.options().dtype(at::kBFloat16));
}
inline Tensor empty_f32(at::IntArrayRef s, const Tensor& like) { return at::empty(s, like.options().dtype(at::kFloat)); }
// A [B, D] modulation tensor whose rows may be strided (a chunk of a wider tensor).
inline Tensor mod_view(const Tensor& t, int64_t D) {
  if (!t.defined()) return t;
  TORCH_CHECK(t.dim() == 2 && t.size(1) == D, "modulation tensor must be [B, ", D, "]");
  return (t.stride(1) != 1 || t.stride(0) % 8 != 0 || !al16(t)) ? t.contiguous() : t;
}

// ---- gemm_ops.cpp
struct GemmOpt {
  Tensor out, bias, lora_h, lora_b, pre_out, pre_in, residual, gate, out2;
  float alpha = 1.f;
  int act = 0, rows_per_batch = 0, n_split = 0, glu = 0;
  bool b_mn = false, a_mn = false, pdl = false;
};
bool gemm_supported(int64_t M, int64_t N, int64_t K);
Tensor gemm(const Tensor& a, const Tensor& b, const GemmOpt& o, int flags);
std::pair<Tensor, Tensor> gemm_pair(const Tensor& a0, const Tensor& b0, const GemmOpt& o0, const Tensor& a1,
                                    const Tensor& b1, const GemmOpt& o1, int flags);
Tensor skinny(const Tensor& a, const Tensor& b, float alpha, int flags);
std::pair<Tensor, Tensor> skinny_pair(const Tensor& a0, const Tensor& b0, float s0, const Tensor& a1, const Tensor& b1,
                                      float s1, int flags);
Tensor wgrad(const Tensor& dy2, const Tensor& x2, const Tensor& accum, int flags);
Tensor lora_wgrad(const Tensor& a_tok, const Tensor& b_tok, Tensor out, bool transpose_out, bool accumulate, int flags);
Tensor lora_transposed(const Tensor& m);
Tensor gate_rows(const Tensor& x, const Tensor& y2, const Tensor& gate, int64_t rows_per_batch);
bool lora_rank_ok(int64_t r);
// Whether p's gradient may be added into p.grad in place (the arena views) instead of being returned for autograd to
// store. ``allowed``: the caller's switch (kAccumGrad).
bool has_grad_buffer(const Tensor& p, at::ScalarType t, bool allowed);

OptT linear(const Tensor& x, const Tensor& w, const OptT& bias, const OptT& la, const OptT& lb, double scale, int act,
            const OptT& residual, const OptT& gate, const OptT& wt, int flags);
std::vector<Tensor> linear_pair(const std::vector<OptT>& s0, double sc0, const std::vector<OptT>& s1, double sc1, int act,
                                bool emit_pre, int act_in, int flags);
Tensor linear_glu(const Tensor& x, const Tensor& w, const OptT& bias, const OptT& la, const OptT& lb, double scale,
                  int code, const OptT& wt, int flags);
Tensor small_linear(const Tensor& x, const Tensor& w, const OptT& bias, bool silu_in, bool accum);
Tensor small_wgrad(const Tensor& dy2, const Tensor& xin, double scale, const Tensor& accum);
Tensor small_dgrad(const Tensor& dy2, const Tensor& w);
int prepare_lora_transposes(const std::vector<Tensor>& mats);
Tensor col_sum(const Tensor& x2, const Tensor& p, bool accum);
void invalidate_lora_transposes(const std::vector<Tensor>& mats);

// ---- block_ops.cpp
std::vector<Tensor> norm_modulate(const Tensor& x, const OptT& scale, const OptT& shift, const OptT& weight,
                                  const OptT& bias, double eps, bool rms, bool skip, bool accum);
std::vector<Tensor> qknorm_rope_joint(const std::vector<OptT>& flat, const OptT& cos, const OptT& sin, int64_t heads,
                                      double eps);
Tensor gate_residual(const OptT& x, const Tensor& y, const OptT& gate);
Tensor act(const Tensor& x, int mode);
Tensor glu(const Tensor& h, int mode, bool act_first);
std::vector<Tensor> split_tokens(const Tensor& x, int64_t n);
Tensor attention(const Tensor& q, const Tensor& k, const Tensor& v, double scale, const OptT& kbias, int pair_poly);
Tensor attention_qkv(const Tensor& qkv, int64_t heads, double scale, const OptT& kbias);
Tensor attention_kv(const Tensor& q, const Tensor& kv, int64_t heads, double scale, const OptT& kbias);
Tensor attention_wide(const Tensor& q, const Tensor& k, const Tensor& v, double scale);
Tensor attention_bias(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& bias, double scale);
Tensor attention_qkv_rope(const Tensor& qkv, const Tensor& wq, const Tensor& wk, const Tensor& cos, const Tensor& sin,
                          int64_t heads, double eps);
Tensor mse_loss(const Tensor& pred, const Tensor& target, const OptT& weight);
Tensor group_norm_silu(const Tensor& x, const Tensor& weight, const OptT& bias, const OptT& pre_c, const OptT& pre_nc,
                       int64_t groups, double eps, bool silu, bool accum);
Tensor add_bias(const Tensor& a, const Tensor& b, const OptT& bias, const OptT& bias2, bool accum);
Tensor upsample2x(const Tensor& x);
Tensor conv2d_trained(const Tensor& x, const Tensor& w, const std::vector<int64_t>& stride, const std::vector<int64_t>& padding,
                      const std::vector<int64_t>& dilation, bool accum);
Tensor single_stream(const Tensor& xm, const Tensor& x, const Tensor& gate, const Tensor& w1, const OptT& b1,
                     const Tensor& w2, const OptT& b2, const OptT& a1, const OptT& bb1, double s1, const OptT& a2,
                     const OptT& bb2, double s2, const OptT& qs, const OptT& ks, const OptT& cos, const OptT& sin,
                     int64_t heads, int flags, bool act_fwd_epilogue, bool act_bwd_epilogue);

// Optional tensors among a node's arguments. Function::apply takes them as std::optional, and only the present ones
// get an edge: ``Args`` records which are present (arguments come first, in order) so that the backward can ask
// for an argument by its position.
inline OptT wrap(const Tensor& t) { return t.defined() ? OptT(t) : OptT(); }
struct Args {
  int64_t mask = 0;
  Args(std::initializer_list<const Tensor*> ts) {
    int i = 0;
    for (const Tensor* t : ts) mask |= (int64_t)t->defined() << i++;
  }
  explicit Args(int64_t m) : mask(m) {}
  bool need(AutogradContext* ctx, int i) const {
    return ((mask >> i) & 1) && ctx->needs_input_grad((size_t)__builtin_popcountll((uint64_t)mask & ((1ull << i) - 1)));
  }
};

// The kernels have no forward-mode derivatives. A dual tensor is refused, whether or not gradients are recorded: its
// result would silently have no tangent.
inline void refuse_tangents(std::initializer_list<const Tensor*> ts) {
  if (!torch::autograd::ForwardADLevel::try_get_by_idx(0)) return;      // no dual level is open
  for (const Tensor* t : ts)
    TORCH_CHECK_NOT_IMPLEMENTED(!t->defined() || !t->_fw_grad(0).defined(), "forward-mode differentiation of this op");
}

// Whether a node is needed for these inputs.
inline bool any_grad(std::initializer_list<const Tensor*> ts) {
  refuse_tangents(ts);
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor* t : ts)
    if (t->defined() && t->requires_grad()) return true;
  return false;
}

}  // namespace eri_ops
