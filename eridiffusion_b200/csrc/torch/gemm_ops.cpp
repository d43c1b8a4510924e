// Matrix products of the op layer: the tensor-core GEMM and its adapter companions, and the autograd nodes of
// the fused linears. Forward and backward of a linear are launch sequences whose order matters: the rank-r
// product of an adapter is the launch right before the GEMM that consumes it, which is then scheduled as its
// programmatic dependent.
#include "eri_ops.h"

#include <torch/csrc/autograd/graph_task.h>
#include <torch/csrc/autograd/variable.h>

#include <mutex>
#include <unordered_map>

namespace eri_ops {

namespace {

struct Built {
  EriGemmArgs g;
  Tensor out;
};

Built build(const Tensor& a, const Tensor& b, const GemmOpt& o) {
  Built r;
  EriGemmArgs& g = r.g;
  memset(&g, 0, sizeof(g));
  const int64_t K = o.a_mn ? a.size(0) : a.size(1), M = o.a_mn ? a.size(1) : a.size(0);
  const int64_t N = o.b_mn ? b.size(1) : b.size(0);
  TORCH_CHECK((o.b_mn ? b.size(0) : b.size(1)) == K && a.stride(1) == 1 && b.stride(1) == 1, "gemm: operand layouts");
  r.out = o.out;
  if (!r.out.defined()) r.out = empty_bf16({M, o.glu ? N / 2 : (o.n_split ? o.n_split : N)}, a);
  g.a = a.data_ptr(); g.b = b.data_ptr();
  g.lda = a.stride(0); g.ldb = b.stride(0);
  g.M = (int)M; g.N = (int)N; g.K = (int)K;
  g.alpha = o.alpha;
  g.out = r.out.data_ptr(); g.ldc = (int)r.out.stride(0);
  g.bias = ptr(o.bias);
  if (o.lora_h.defined()) {
    g.lora_h = o.lora_h.data_ptr(); g.lora_b = o.lora_b.data_ptr();
    g.ld_h = o.lora_h.stride(0); g.ld_lb = o.lora_b.stride(0);
    g.lora_r = (int)o.lora_h.size(1);
  }
  g.act = o.act;
  if (o.pre_out.defined()) { g.pre_out = o.pre_out.data_ptr(); g.ld_pre = (int)o.pre_out.stride(0); }
  if (o.pre_in.defined()) { g.pre_in = o.pre_in.data_ptr(); g.ld_pre = (int)o.pre_in.stride(0); }
  if (o.residual.defined()) { g.residual = o.residual.data_ptr(); g.ldr = (int)o.residual.stride(0); }
  if (o.gate.defined()) { g.gate = o.gate.data_ptr(); g.gate_stride = (int)o.gate.stride(0); }
  g.rows_per_batch = o.rows_per_batch;
  g.n_split = o.n_split;
  if (o.out2.defined()) { g.out2 = o.out2.data_ptr(); g.ldc2 = (int)o.out2.stride(0); }
  g.dbg_out_bytes = extent(r.out); g.dbg_out2_bytes = extent(o.out2);
  g.dbg_pre_bytes = extent(o.pre_out); g.dbg_res_bytes = extent(o.residual);
  g.b_mn = o.b_mn; g.a_mn = o.a_mn; g.glu = o.glu;
  g.pdl = o.pdl && o.lora_h.defined();
  return r;
}

// The choice of kernel, as in ops/functional.py: _launch_gemm.
void launch(const EriGemmArgs& g, int flags) {
  // Few 128 x 128 tiles: the K range over a cluster, two CTAs per SM (answers -30 for any other product).
  if (!g.a_mn || (g.M >= 256 && g.N >= 256)) {
    const int code = L.eri_gemm_few_bf16(&g, stream());
    if (code != -30) return check(code, "gemm_few_bf16");
  }
  // Few pair tiles (the 512-token text stream against a 3072-wide weight: 24 tiles for 74 CTA pairs) leave
  // most SMs idle; the one-CTA kernel's 128-column tiles spread the same work over four times as many CTAs.
  const bool few = !(g.a_mn || g.glu) &&
                   (int64_t)((g.M + 255) / 256) * ((g.N + 255) / 256) <= (flags >> kFewTilesShift);
  if (((flags & kPair) || g.a_mn || g.glu) && g.M >= 256 && g.N >= 256 && !few) {
    const int code = L.eri_gemm2_bf16(&g, stream());
    if (code != -30) return check(code, "gemm2_bf16");
  }
  TORCH_CHECK(!(g.a_mn || g.glu), "gemm: a_mn / glu need the two-CTA kernel's shape range (M=", g.M, ", N=", g.N,
              ", K=", g.K, ")");
  check(L.eri_gemm_bf16(&g, stream()), "gemm_bf16");
}

Tensor undef() { return Tensor(); }

}  // namespace

bool gemm_supported(int64_t M, int64_t N, int64_t K) { return M >= 128 && N >= 16 && K >= 8 && K % 8 == 0 && N % 8 == 0; }
bool lora_rank_ok(int64_t r) { return r == 16 || r == 32 || r == 64; }
bool has_grad_buffer(const Tensor& p, at::ScalarType t, bool allowed) {
  if (!allowed || !p.is_leaf() || !p.requires_grad()) return false;
  // torch.autograd.grad and backward(inputs=...) want the gradient itself, and so does whoever hooked the parameter
  const auto* asked = torch::autograd::get_current_graph_task_exec_info();
  if (asked && !asked->empty()) return false;
  if (!torch::autograd::impl::hooks(p).empty() || torch::autograd::impl::post_acc_grad_hooks(p)) return false;
  const Tensor& g = p.grad();
  return g.defined() && g.scalar_type() == t && g.is_contiguous();
}

Tensor gemm(const Tensor& a, const Tensor& b, const GemmOpt& o, int flags) {
  Built r = build(a, b, o);
  launch(r.g, flags);
  return r.out;
}

// Two independent products in one launch of the two-CTA kernel when they qualify, else one after the other.
std::pair<Tensor, Tensor> gemm_pair(const Tensor& a0, const Tensor& b0, const GemmOpt& o0, const Tensor& a1,
                                    const Tensor& b1, const GemmOpt& o1, int flags) {
  Built r0 = build(a0, b0, o0), r1 = build(a1, b1, o1);
  const EriGemmArgs &g0 = r0.g, &g1 = r1.g;
  const bool plain = g0.M >= 256 && g0.N >= 256 && g1.M >= 256 && g1.N >= 256 && !(g0.a_mn || g0.glu || g1.a_mn || g1.glu);
  if ((flags & kGroup) && (flags & kPair) && plain) {
    const int code = L.eri_gemm2_bf16_group2(&g0, &g1, stream());
    if (code != -30) {
      check(code, "gemm2_bf16_group2");
      return {r0.out, r1.out};
    }
  }
  launch(g0, flags);
  launch(g1, flags);
  return {r0.out, r1.out};
}

// alpha * a[M, K] @ b[N, K]^T for N = an adapter rank.
Tensor skinny(const Tensor& a, const Tensor& b, float alpha, int flags) {
  const int64_t M = a.size(0), K = a.size(1), N = b.size(0);
  if (a.stride(1) == 1 && b.stride(1) == 1) {
    Tensor out = empty_bf16({M, N}, a);
    if (flags & kRankStream) {
      const int code = L.eri_gemm_rank_stream(a.data_ptr(), a.stride(0), b.data_ptr(), b.stride(0), out.data_ptr(),
                                              (int)N, (int)M, (int)N, (int)K, alpha, stream());
      if (code != -100) return check(code, "gemm_rank_stream"), out;
    }
    if (M >= 128) {
      const int code = L.eri_gemm_skinny(a.data_ptr(), a.stride(0), b.data_ptr(), b.stride(0), out.data_ptr(), (int)N,
                                         (int)M, (int)N, (int)K, alpha, stream());
      if (code != -100) return check(code, "gemm_skinny"), out;
    }
  }
  GemmOpt o;
  o.alpha = alpha;
  return gemm(a, b, o, flags);
}

std::pair<Tensor, Tensor> skinny_pair(const Tensor& a0, const Tensor& b0, float s0, const Tensor& a1, const Tensor& b1,
                                      float s1, int flags) {
  if ((flags & kRankStream) && (flags & kGroup) && a0.size(1) == a1.size(1) && b0.size(0) == b1.size(0) &&
      a0.stride(1) == 1 && b0.stride(1) == 1 && a1.stride(1) == 1 && b1.stride(1) == 1) {
    const int r = (int)b0.size(0), K = (int)a0.size(1);
    Tensor h0 = empty_bf16({a0.size(0), r}, a0), h1 = empty_bf16({a1.size(0), r}, a1);
    const int code = L.eri_gemm_rank_stream2(
        a0.data_ptr(), a0.stride(0), b0.data_ptr(), b0.stride(0), h0.data_ptr(), r, (int)a0.size(0), s0, a1.data_ptr(),
        a1.stride(0), b1.data_ptr(), b1.stride(0), h1.data_ptr(), r, (int)a1.size(0), s1, r, K, stream());
    if (code != -100) {
      check(code, "gemm_rank_stream2");
      return {h0, h1};
    }
  }
  Tensor h0 = skinny(a0, b0, s0, flags);
  return {h0, skinny(a1, b1, s1, flags)};
}

// dW[N, K] = dy2[T, N]^T x2[T, K]; ``accum``: added into it (beta = 1 in the epilogue).
Tensor wgrad(const Tensor& dy2, const Tensor& x2, const Tensor& accum, int flags) {
  const int64_t T = dy2.size(0), N = dy2.size(1), K = x2.size(1);
  const bool native = (flags & kWgrad) && (flags & kNativeGemm) && rows_ok(dy2) && rows_ok(x2) && N >= 256 && K >= 256 &&
                      T >= 64 && N % 8 == 0 && K % 8 == 0 && (!accum.defined() || rows_ok(accum));
  if (native) {
    GemmOpt o;
    o.a_mn = o.b_mn = true;
    o.out = o.residual = accum;
    return gemm(dy2, x2, o, flags);
  }
  if (accum.defined()) {
    Tensor acc = accum;
    return acc.addmm_(dy2.t(), x2);
  }
  return at::mm(dy2.t(), x2);
}

// Adapter gradients a_tok[T, Mg]^T b_tok[T, r] ([r, Mg] with transpose_out), optionally added into ``out``.
Tensor lora_wgrad(const Tensor& a_tok, const Tensor& b_tok, Tensor out, bool transpose_out, bool accumulate, int flags) {
  const int64_t T = a_tok.size(0), Mg = a_tok.size(1), r = b_tok.size(1);
  const int64_t d0 = transpose_out ? r : Mg, d1 = transpose_out ? Mg : r;
  if ((flags & kWgrad) && (flags & kNativeGemm) && rows_ok(a_tok) && lora_rank_ok(r) && rows_ok(b_tok) && T >= 64 &&
      Mg >= 128 && Mg % 8 == 0 &&
      (!out.defined() || (out.scalar_type() == at::kBFloat16 && out.stride(1) == 1 && out.size(0) == d0 && out.size(1) == d1))) {
    if (!out.defined()) {
      out = empty_bf16({d0, d1}, a_tok);
      accumulate = false;
    }
    const int code = L.eri_gemm_tokred(a_tok.data_ptr(), a_tok.stride(0), b_tok.data_ptr(), b_tok.stride(0), out.data_ptr(),
                                       (int)out.stride(0), (int)T, (int)Mg, (int)r, 1.f, transpose_out, accumulate,
                                       extent(out), stream());
    if (code != -100) return check(code, "gemm_tokred"), out;
  }
  Tensor prod = transpose_out ? at::mm(b_tok.t(), a_tok) : at::mm(a_tok.t(), b_tok);
  if (!out.defined()) return prod;
  return accumulate ? out.add_(prod) : out.copy_(prod);
}

Tensor gate_rows(const Tensor& x, const Tensor& y2, const Tensor& gate, int64_t rows_per_batch) {
  Tensor g = at::empty_like(y2);
  check(L.eri_gate_residual(ptr(x), y2.data_ptr(), gate.data_ptr(), g.data_ptr(), y2.size(0), (int)y2.size(1),
                            (int)rows_per_batch, (int)gate.stride(0), stream()), "gate_residual");
  return g;
}

// ------------------------------------------------------------------------------- transposed adapter matrices
// The backward of an adapted linear reads B^T and A^T. One launch per optimizer step transposes every adapter
// matrix of a model; a plan (destination buffer + job list on the device) belongs to one set of matrices and
// is dropped when they are gone. Without a valid copy the two small matrices are transposed at the site.
namespace {
struct TransposeJob {
  const void* src;
  void* dst;
  int rows, cols;
};
struct TransposePlan {
  std::vector<void*> key;
  std::vector<c10::weak_intrusive_ptr<c10::TensorImpl>> owners;
  std::vector<Tensor> outs;
  Tensor buf, jobs;
  int64_t max_elems = 0;
  bool valid = false;
  // matrix i is still the tensor it was made from, at the same address
  bool current(size_t i) const {
    const auto t = owners[i].lock();
    return t && t->data() == key[i];
  }
};
std::mutex g_tmu;
std::vector<std::shared_ptr<TransposePlan>> g_plans;
std::unordered_map<void*, std::pair<std::weak_ptr<TransposePlan>, int>> g_published;

constexpr size_t kMaxPlans = 64;     // models that train side by side in one process

void drop_plan(size_t i) {
  for (void* k : g_plans[i]->key) {
    auto it = g_published.find(k);
    if (it != g_published.end() && it->second.first.lock() == g_plans[i]) g_published.erase(it);
  }
  g_plans.erase(g_plans.begin() + (long)i);
}
void drop_dead_plans() {
  for (size_t i = g_plans.size(); i-- > 0;)
    for (size_t j = 0; j < g_plans[i]->key.size(); ++j)
      if (!g_plans[i]->current(j)) {
        drop_plan(i);
        break;
      }
  while (g_plans.size() >= kMaxPlans) drop_plan(0);
}
}  // namespace

int prepare_lora_transposes(const std::vector<Tensor>& all) {
  std::vector<Tensor> mats;
  for (const Tensor& m : all)
    if (m.is_cuda() && m.scalar_type() == at::kBFloat16 && m.dim() == 2 && m.is_contiguous()) mats.push_back(m);
  if (mats.empty()) return 0;
  std::vector<void*> key;
  key.reserve(mats.size());
  for (const Tensor& m : mats) key.push_back(m.data_ptr());
  std::lock_guard<std::mutex> lock(g_tmu);
  drop_dead_plans();
  std::shared_ptr<TransposePlan> plan;
  for (auto& p : g_plans)
    if (p->key == key) plan = p;
  if (!plan) {
    plan = std::make_shared<TransposePlan>();
    plan->key = key;
    int64_t total = 0;
    for (const Tensor& m : mats) total += m.numel();
    plan->buf = empty_bf16({total}, mats[0]);
    std::vector<TransposeJob> jobs(mats.size());
    int64_t off = 0;
    for (size_t i = 0; i < mats.size(); ++i) {
      const Tensor& m = mats[i];
      Tensor o = plan->buf.narrow(0, off, m.numel()).view({m.size(1), m.size(0)});
      jobs[i] = {m.data_ptr(), o.data_ptr(), (int)m.size(0), (int)m.size(1)};
      plan->outs.push_back(o);
      plan->owners.emplace_back(m.getIntrusivePtr());
      plan->max_elems = std::max(plan->max_elems, m.numel());
      off += m.numel();
    }
    Tensor host = at::empty({(int64_t)(jobs.size() * sizeof(TransposeJob))}, at::TensorOptions().dtype(at::kByte));
    memcpy(host.data_ptr(), jobs.data(), jobs.size() * sizeof(TransposeJob));
    plan->jobs = host.to(mats[0].device());
    g_plans.push_back(plan);
    for (size_t i = 0; i < key.size(); ++i) g_published[key[i]] = {plan, (int)i};
  }
  check(L.eri_batched_transpose(plan->jobs.data_ptr(), (int)mats.size(), (int)plan->max_elems, stream()), "batched_transpose");
  plan->valid = true;
  return (int)mats.size();
}

// The matrices changed (optimizer step): the copies of every plan that one of them is published by are stale. With an
// empty list every plan is.
void invalidate_lora_transposes(const std::vector<Tensor>& mats) {
  std::lock_guard<std::mutex> lock(g_tmu);
  if (mats.empty()) {
    for (auto& p : g_plans) p->valid = false;
    return;
  }
  for (const Tensor& m : mats) {
    auto it = g_published.find(m.data_ptr());
    if (it == g_published.end()) continue;
    if (auto p = it->second.first.lock()) p->valid = false;
  }
}

Tensor lora_transposed(const Tensor& m) {
  {
    std::lock_guard<std::mutex> lock(g_tmu);
    auto it = g_published.find(m.data_ptr());
    if (it != g_published.end()) {
      auto p = it->second.first.lock();
      const int i = it->second.second;
      if (p && p->valid && p->current(i) && p->outs[i].size(0) == m.size(1) && p->outs[i].size(1) == m.size(0))
        return p->outs[i];
    }
  }
  return m.t().contiguous();
}

// Column sums of x2 [M, N] for the parameter p (a bias): added straight into p.grad when it has a buffer of that
// type (an undefined tensor is returned then), else returned.
Tensor col_sum(const Tensor& x2, const Tensor& p, bool accum) {
  const bool acc = has_grad_buffer(p, x2.scalar_type(), accum);
  if (x2.size(0) > 0 && rows_ok(x2) && x2.size(1) % 8 == 0 && (!acc || al16(p.grad()))) {
    Tensor out = acc ? p.grad() : empty_bf16({x2.size(1)}, x2);
    check(L.eri_col_sum(x2.data_ptr(), x2.stride(0), out.data_ptr(), (int)x2.size(0), (int)x2.size(1), acc, stream()),
          "col_sum");
    return acc ? undef() : out;
  }
  return x2.sum(0);
}

// ------------------------------------------------------------------------------------------ fused linear
namespace {

Tensor activation(const Tensor& y, int act) { return act == 1 ? at::gelu(y, "tanh") : at::silu(y); }

// [x +] gate * y for row widths the vector kernel does not take
Tensor gate_rows_any(const Tensor& x, const Tensor& y2, const Tensor& gate, int64_t rows_per_batch) {
  const int64_t N = y2.size(1);
  Tensor o = y2.view({-1, rows_per_batch, N}).to(at::kFloat) * gate.to(at::kFloat).unsqueeze(1);
  if (x.defined()) o = o + x.view({-1, rows_per_batch, N}).to(at::kFloat);
  return o.to(y2.scalar_type()).view({-1, N});
}

struct LinGrads {
  Tensor dx, dw, db, da, dlb;
};

// Gradients of y = x W^T + b + s (x A^T) B^T given dy2 = dL/dy [M, N].
LinGrads linear_grads(const Tensor& dy2, const Tensor& x2, const Tensor& w, const Tensor& bias, const Tensor& la,
                      const Tensor& lb, const Tensor& h, float s, const Tensor& wt, bool nx, bool nw, bool nb, bool na,
                      bool nlb, at::IntArrayRef shp, int flags) {
  LinGrads g;
  const int64_t M = x2.size(0), K = x2.size(1), N = dy2.size(1);
  const int64_t r = la.defined() ? la.size(0) : 0;
  const bool native = (flags & kNativeGemm) && gemm_supported(M, K, N);
  Tensor ts, la_t;
  if (r) {
    if (native && lora_rank_ok(r)) {
      // both transposes are looked up first: nothing may launch between Ts and the dX GEMM
      Tensor lb_t = lora_transposed(lb);
      la_t = lora_transposed(la);
      ts = skinny(dy2, lb_t, s, flags);
    } else {
      ts = at::mm(dy2, lb).mul_(s);
    }
  }
  if (nx) {
    if (native) {
      // dX = dY W: W itself is the MN-major operand (no copy), or a cached transpose of it the K-major one
      GemmOpt o;
      Tensor b_op = wt.defined() ? wt : w;
      o.b_mn = !wt.defined();
      const bool copied = o.b_mn && K < 64;
      if (copied) {
        b_op = w.t().contiguous();       // a launch between Ts and the GEMM
        o.b_mn = false;
      }
      if (lora_rank_ok(r)) {
        o.lora_h = ts;
        o.lora_b = la_t;
        o.pdl = (flags & kPdl) && !copied;
      }
      g.dx = gemm(dy2, b_op, o, flags);
      if (r && !lora_rank_ok(r)) g.dx = g.dx + at::mm(ts, la);
    } else {
      g.dx = at::mm(dy2, w);
      if (r) g.dx = g.dx + at::mm(ts, la);
    }
    g.dx = g.dx.view(shp);
  }
  if (nw) {
    if (has_grad_buffer(w, x2.scalar_type(), flags & kAccumGrad))
      wgrad(dy2, x2, w.grad(), flags);       // beta = 1 into the (arena) gradient view
    else
      g.dw = wgrad(dy2, x2, Tensor(), flags);
  }
  if (nb) g.db = col_sum(dy2, bias, flags & kAccumGrad);
  if (r && na) {
    if (has_grad_buffer(la, x2.scalar_type(), flags & kAccumGrad))
      lora_wgrad(x2, ts, la.grad(), true, true, flags);
    else
      g.da = lora_wgrad(x2, ts, Tensor(), true, false, flags);
  }
  if (r && nlb) {
    if (has_grad_buffer(lb, h.scalar_type(), flags & kAccumGrad))
      lora_wgrad(dy2, h, lb.grad(), false, true, flags);
    else
      g.dlb = lora_wgrad(dy2, h, Tensor(), false, false, flags);
  }
  return g;
}

Tensor act_bwd(const Tensor& dy2, const Tensor& pre, int act) {
  if (dy2.numel() % 8) return act == 1 ? at::gelu_backward(dy2, pre, "tanh") : at::silu_backward(dy2, pre);
  Tensor g = at::empty_like(dy2);
  check(L.eri_act_bwd(dy2.data_ptr(), pre.data_ptr(), g.data_ptr(), dy2.numel(), act - 1, stream()), "act_bwd");
  return g;
}
Tensor act_fwd(const Tensor& pre, int act) {
  Tensor y = at::empty_like(pre);
  check(L.eri_act_fwd(pre.data_ptr(), y.data_ptr(), pre.numel(), act - 1, stream()), "act_fwd");
  return y;
}

struct LinOut {
  Tensor y, x2, h, pre, gate;
};

// y = [residual + gate *] act(x W^T + b + s (x A^T) B^T), M = B * L rows. ``keep``: a gradient will be asked for.
LinOut linear_forward(const Tensor& x, const Tensor& w, const Tensor& bias, const Tensor& la, const Tensor& lb,
                      const Tensor& residual, const Tensor& gate, float s, int act, bool keep, int flags) {
  LinOut r;
  const int64_t K = x.size(-1), N = w.size(0), L_ = x.dim() >= 2 ? x.size(-2) : 1;
  r.x2 = contig(x).view({-1, K});
  const int64_t M = r.x2.size(0);
  const int64_t rank = la.defined() ? la.size(0) : 0;
  const bool native = (flags & kNativeGemm) && gemm_supported(M, N, K);
  Tensor res2 = residual.defined() ? contig(residual).view({-1, N}) : residual;
  r.gate = mod_view(gate, N);
  Tensor y;
  if (native && (!rank || lora_rank_ok(rank))) {
    GemmOpt o;
    o.bias = bias;
    o.pdl = flags & kPdl;
    if (act && keep) r.pre = empty_bf16({M, N}, x);
    const bool split = r.pre.defined() && !res2.defined() && !r.gate.defined() && (flags & kActOutside);
    if (split) {
      // training keeps the pre-activation anyway: the GEMM writes it as its output and the activation is a pass
      // of its own (cheaper than storing both from the epilogue)
      o.out = r.pre;
    } else {
      o.act = act;
      o.pre_out = r.pre;
      o.residual = res2;
      o.gate = r.gate;
      o.rows_per_batch = (int)L_;
      o.out = empty_bf16({M, N}, x);
    }
    if (rank) {
      r.h = o.lora_h = skinny(r.x2, la, s, flags);     // the launch right before the GEMM
      o.lora_b = lb;
    }
    y = gemm(r.x2, w, o, flags);
    if (split) y = act_fwd(r.pre, act);
  } else {
    if (native) {
      GemmOpt o;
      o.bias = bias;
      r.h = at::mm(r.x2, la.t()).mul_(s);
      y = gemm(r.x2, w, o, flags) + at::mm(r.h, lb.t());
    } else {
      y = bias.defined() ? at::linear(r.x2, w, bias) : at::linear(r.x2, w);
      if (rank) {
        r.h = at::mm(r.x2, la.t()).mul_(s);
        y = y + at::mm(r.h, lb.t());
      }
    }
    if (act) {
      r.pre = y;
      y = activation(y, act);
    }
    if (r.gate.defined()) {
      y = N % 8 == 0 ? gate_rows(res2, contig(y), r.gate, L_) : gate_rows_any(res2, y, r.gate, L_);
    } else if (res2.defined()) {
      y = y + res2;
    }
  }
  auto shp = x.sizes().vec();
  shp.back() = N;
  r.y = y.view(shp);
  return r;
}

struct FusedLinear : torch::autograd::Function<FusedLinear> {
  static Tensor forward(AutogradContext* ctx, const OptT& x_o, const OptT& w_o, const OptT& bias_o, const OptT& la_o,
                        const OptT& lb_o, const OptT& residual_o, const OptT& gate_o, const OptT& wt_o, double s,
                        int64_t act, int64_t flags) {
    const Tensor x = opt(x_o), w = opt(w_o), bias = opt(bias_o), la = opt(la_o), lb = opt(lb_o), residual = opt(residual_o), gate = opt(gate_o), wt = opt(wt_o);
    if (ctx) ctx->saved_data["args"] = Args({&x, &w, &bias, &la, &lb, &residual, &gate, &wt}).mask;
    LinOut r = linear_forward(x, w, bias, la, lb, residual, gate, (float)s, (int)act, true, (int)flags);
    ctx->save_for_backward({r.x2, w, bias, la, lb, r.h, r.pre, r.gate, wt});
    ctx->saved_data["s"] = s;
    ctx->saved_data["m"] = std::vector<int64_t>{act, flags, residual.defined(), x.dim() >= 2 ? x.size(-2) : 1};
    ctx->saved_data["shp"] = x.sizes().vec();
    return r.y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list gout) {
    auto sv = ctx->get_saved_variables();
    const Tensor &x2 = sv[0], &w = sv[1], &bias = sv[2], &la = sv[3], &lb = sv[4], &h = sv[5], &pre = sv[6], &gate = sv[7];
    const auto m = ctx->saved_data["m"].toIntVector();
    const auto shp = ctx->saved_data["shp"].toIntVector();
    const int act = (int)m[0], flags = (int)m[1];
    const Tensor& dy = gout[0];
    const int64_t M = x2.size(0), N = w.size(0);
    Tensor dy2 = contig(dy).view({M, N});
    if (gate.defined()) dy2 = N % 8 == 0 ? gate_rows(Tensor(), dy2, gate, m[3]) : gate_rows_any(Tensor(), dy2, gate, m[3]);
    if (act) dy2 = act_bwd(dy2, pre, act);
    const Args args(ctx->saved_data["args"].toInt());
    auto need = [&](int i) { return args.need(ctx, i); };
    LinGrads g = linear_grads(dy2, x2, w, bias, la, lb, h, (float)ctx->saved_data["s"].toDouble(), sv[8], need(0), need(1),
                              need(2), need(3), need(4), shp, flags);
    return {g.dx, g.dw, g.db, g.da, g.dlb, m[2] ? dy : Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

}  // namespace

// nullopt: the operands are not on the native path (dtype, device, width) and the caller takes its own.
OptT linear(const Tensor& x, const Tensor& w, const OptT& bias_, const OptT& la_, const OptT& lb_, double scale, int act,
            const OptT& residual_, const OptT& gate_, const OptT& wt_, int flags) {
  Tensor bias = opt(bias_), la = opt(la_), lb = opt(lb_), residual = opt(residual_), gate = opt(gate_), wt = opt(wt_);
  if (!bf16_cuda(x) || !bf16_cuda(w) || !bf16_cuda(bias) || x.size(-1) % 8) return std::nullopt;
  if (gate.defined() && any_grad({&gate})) {
    // trainable modulation: the gate stays outside the GEMM epilogue so that its gradient is produced
    OptT y = linear(x, w, bias_, la_, lb_, scale, act, std::nullopt, std::nullopt, wt_, flags);
    return gate_residual(residual_, *y, gate_);
  }
  if (any_grad({&x, &w, &bias, &la, &lb, &residual}))
    return FusedLinear::apply(wrap(x), wrap(w), wrap(bias), wrap(la), wrap(lb), wrap(residual), wrap(gate), wrap(wt), scale, (int64_t)act, (int64_t)flags);
  return linear_forward(x, w, bias, la, lb, residual, gate, (float)scale, act, false, flags).y;
}

// ------------------------------------------------------------------------------------- pair of linears
// Two fused linears with the same shape of weight (the image and the text stream of a dual-stream block): the
// two main GEMMs share one launch in the forward and the two input-gradient GEMMs one in the backward, as do
// the rank-r products of both streams; everything else is what FusedLinear does per stream.
//
// Two more modes chain an MLP without a separate activation-gradient pass. ``emit_pre``: the outputs are
// (pre_0, pre_1, u_0, u_1) with u_i = act(pre_i) marked non-differentiable, i.e. the layer is the plain linear
// that produces the pre-activation and the activation is a by-product of its epilogue. ``act_in`` with xp_i:
// x_i is act_in(xp_i) (such a by-product), the layer is linear-of-activation as a function of xp_i, and its
// input-gradient GEMM applies the activation's derivative at xp_i in its epilogue.
namespace {

struct Stream {       // positions of a stream's tensors among the node's arguments
  enum { x = 0, xp, w, b, la, lb, res, gate, kCount };
};

struct FusedLinearPair : torch::autograd::Function<FusedLinearPair> {
  static variable_list forward(AutogradContext* ctx, const OptT& x0_o, const OptT& xp0_o, const OptT& w0_o, const OptT& b0_o,
                               const OptT& la0_o, const OptT& lb0_o, const OptT& res0_o, const OptT& gate0_o,
                               const OptT& x1_o, const OptT& xp1_o, const OptT& w1_o, const OptT& b1_o, const OptT& la1_o,
                               const OptT& lb1_o, const OptT& res1_o, const OptT& gate1_o, double s0, double s1, int64_t act,
                               bool emit_pre, int64_t act_in, int64_t keep0, int64_t keep1, int64_t flags) {
    const Tensor x0 = opt(x0_o), xp0 = opt(xp0_o), w0 = opt(w0_o), b0 = opt(b0_o), la0 = opt(la0_o), lb0 = opt(lb0_o), res0 = opt(res0_o), gate0 = opt(gate0_o), x1 = opt(x1_o), xp1 = opt(xp1_o), w1 = opt(w1_o), b1 = opt(b1_o), la1 = opt(la1_o), lb1 = opt(lb1_o), res1 = opt(res1_o), gate1 = opt(gate1_o);
    if (ctx) ctx->saved_data["args"] = Args({&x0, &xp0, &w0, &b0, &la0, &lb0, &res0, &gate0, &x1, &xp1, &w1, &b1, &la1, &lb1, &res1, &gate1}).mask;
    const Tensor* in[2][8] = {{&x0, &xp0, &w0, &b0, &la0, &lb0, &res0, &gate0}, {&x1, &xp1, &w1, &b1, &la1, &lb1, &res1, &gate1}};
    const double sc[2] = {s0, s1};
    const bool keep[2] = {keep0 != 0, keep1 != 0};
    GemmOpt o[2];
    Tensor x2[2], h[2], pre[2], gv[2], xp2[2];
    int64_t N[2], M[2], K[2], Lr[2];
    for (int i = 0; i < 2; ++i) {
      const Tensor &x = *in[i][Stream::x], &w = *in[i][Stream::w];
      K[i] = x.size(-1); N[i] = w.size(0); Lr[i] = x.size(-2);
      x2[i] = contig(x).view({-1, K[i]});
      M[i] = x2[i].size(0);
      if (act && (keep[i] || emit_pre)) pre[i] = empty_bf16({M[i], N[i]}, x);
      gv[i] = mod_view(*in[i][Stream::gate], N[i]);
      if (in[i][Stream::xp]->defined()) xp2[i] = contig(*in[i][Stream::xp]).view({-1, K[i]});
      o[i].bias = *in[i][Stream::b];
      if (in[i][Stream::res]->defined()) o[i].residual = contig(*in[i][Stream::res]).view({-1, N[i]});
      o[i].gate = gv[i];
      o[i].rows_per_batch = (int)Lr[i];
      o[i].act = (int)act;
      o[i].pre_out = pre[i];
      o[i].pdl = flags & kPdl;
    }
    // Training keeps the pre-activation anyway: the GEMM then writes it as its output and the activation is a
    // pass of its own (storing both from the epilogue costs the GEMM more than that pass does).
    bool unfuse = act && (flags & kActOutside);
    for (int i = 0; i < 2; ++i) unfuse = unfuse && pre[i].defined() && !o[i].residual.defined() && !gv[i].defined();
    for (int i = 0; i < 2; ++i) {
      if (unfuse) {
        o[i].out = pre[i];
        o[i].act = 0;
        o[i].pre_out = Tensor();
      } else {
        o[i].out = empty_bf16({M[i], N[i]}, x2[i]);
      }
    }
    if (la0.defined()) {
      // both rank-r products in one launch, right before the grouped GEMM that consumes them
      std::tie(h[0], h[1]) = skinny_pair(x2[0], la0, (float)sc[0], x2[1], la1, (float)sc[1], (int)flags);
      for (int i = 0; i < 2; ++i) {
        o[i].lora_h = h[i];
        o[i].lora_b = *in[i][Stream::lb];
      }
    }
    auto [y0, y1] = gemm_pair(x2[0], w0, o[0], x2[1], w1, o[1], (int)flags);
    Tensor y[2] = {y0, y1};
    if (unfuse)
      for (int i = 0; i < 2; ++i) y[i] = act_fwd(pre[i], (int)act);
    ctx->save_for_backward({x2[0], w0, b0, la0, lb0, h[0], emit_pre ? Tensor() : pre[0], gv[0], xp2[0],
                            x2[1], w1, b1, la1, lb1, h[1], emit_pre ? Tensor() : pre[1], gv[1], xp2[1]});
    ctx->saved_data["m"] = std::vector<int64_t>{act, emit_pre, act_in, flags, Lr[0], Lr[1], res0.defined(), res1.defined()};
    ctx->saved_data["s"] = std::vector<double>{s0, s1};
    ctx->saved_data["shp0"] = x0.sizes().vec();
    ctx->saved_data["shp1"] = x1.sizes().vec();
    ctx->set_materialize_grads(false);       // an unused output (undefined gradient) costs nothing in backward
    auto shape_of = [](const Tensor& x, int64_t n) {
      auto s = x.sizes().vec();
      s.back() = n;
      return s;
    };
    const auto ys0 = shape_of(x0, N[0]), ys1 = shape_of(x1, N[1]);
    y[0] = y[0].view(ys0);
    y[1] = y[1].view(ys1);
    if (emit_pre) {
      ctx->mark_non_differentiable({y[0], y[1]});
      return {pre[0].view(ys0), pre[1].view(ys1), y[0], y[1]};
    }
    return {y[0], y[1]};
  }

  static variable_list backward(AutogradContext* ctx, variable_list gout) {
    auto sv = ctx->get_saved_variables();
    const auto m = ctx->saved_data["m"].toIntVector();
    const auto sc = ctx->saved_data["s"].toDoubleVector();
    const int act = (int)m[0], act_in = (int)m[2], flags = (int)m[3];
    const bool emit_pre = m[1];
    const std::vector<int64_t> shp[2] = {ctx->saved_data["shp0"].toIntVector(), ctx->saved_data["shp1"].toIntVector()};
    Tensor dy2[2], ts[2], lbt[2], lat[2];
    bool live[2], want[2];
    GemmOpt o[2];
    const Args args(ctx->saved_data["args"].toInt());
    auto need = [&](int i, int pos) { return args.need(ctx, i * Stream::kCount + pos); };
    for (int i = 0; i < 2; ++i) {
      const Tensor* t = &sv[9 * i];      // x2 w b la lb h pre gate xp
      live[i] = gout[i].defined();
      want[i] = live[i] && need(i, act_in ? Stream::xp : Stream::x);
      if (!live[i]) continue;
      dy2[i] = contig(gout[i]).view({t[0].size(0), t[1].size(0)});
      if (t[7].defined()) dy2[i] = gate_rows(Tensor(), dy2[i], t[7], m[4 + i]);
      if (act && !emit_pre) dy2[i] = act_bwd(dy2[i], t[6], act);
      if (t[3].defined()) {
        lbt[i] = lora_transposed(t[4]);
        lat[i] = lora_transposed(t[3]);
      }
      o[i].b_mn = true;
      o[i].lora_b = lat[i];
      o[i].pdl = flags & kPdl;
      if (act_in) {      // the input's activation derivative in the epilogue
        o[i].act = act_in + 2;
        o[i].pre_in = t[8];
      }
    }
    // Ts_i = s_i * dY_i B_i: one launch for both streams when both have a gradient, right before the grouped
    // input-gradient GEMM
    const bool adapters = sv[3].defined();
    if (adapters && live[0] && live[1]) {
      std::tie(ts[0], ts[1]) = skinny_pair(dy2[0], lbt[0], (float)sc[0], dy2[1], lbt[1], (float)sc[1], flags);
    } else if (adapters) {
      for (int i = 0; i < 2; ++i)
        if (live[i]) ts[i] = skinny(dy2[i], lbt[i], (float)sc[i], flags);
    }
    for (int i = 0; i < 2; ++i) o[i].lora_h = ts[i];
    Tensor dx[2];
    if (want[0] && want[1]) {
      std::tie(dx[0], dx[1]) = gemm_pair(dy2[0], sv[1], o[0], dy2[1], sv[10], o[1], flags);
    } else {
      for (int i = 0; i < 2; ++i)
        if (want[i]) dx[i] = gemm(dy2[i], sv[9 * i + 1], o[i], flags);
    }
    variable_list out(2 * Stream::kCount + 8);
    for (int i = 0; i < 2; ++i) {
      if (!live[i]) continue;
      const Tensor *t = &sv[9 * i], &x2 = t[0], &w = t[1], &la = t[3], &lb = t[4], &h = t[5];
      Tensor* g = &out[i * Stream::kCount];
      if (need(i, Stream::w)) {
        if (has_grad_buffer(w, x2.scalar_type(), flags & kAccumGrad))
          wgrad(dy2[i], x2, w.grad(), flags);
        else
          g[Stream::w] = wgrad(dy2[i], x2, Tensor(), flags);
      }
      if (need(i, Stream::b)) g[Stream::b] = col_sum(dy2[i], t[2], flags & kAccumGrad);
      if (need(i, Stream::la)) {
        if (has_grad_buffer(la, x2.scalar_type(), flags & kAccumGrad))
          lora_wgrad(x2, ts[i], la.grad(), true, true, flags);
        else
          g[Stream::la] = lora_wgrad(x2, ts[i], Tensor(), true, false, flags);
      }
      if (need(i, Stream::lb)) {
        if (has_grad_buffer(lb, h.scalar_type(), flags & kAccumGrad))
          lora_wgrad(dy2[i], h, lb.grad(), false, true, flags);
        else
          g[Stream::lb] = lora_wgrad(dy2[i], h, Tensor(), false, false, flags);
      }
      if (dx[i].defined()) g[act_in ? Stream::xp : Stream::x] = dx[i].view(shp[i]);
      if (m[6 + i]) g[Stream::res] = gout[i];
    }
    return out;
  }
};

}  // namespace

// s0 / s1: [x, xp, w, bias, lora_A, lora_B, residual, gate] of a stream.
std::vector<Tensor> linear_pair(const std::vector<OptT>& s0, double sc0, const std::vector<OptT>& s1, double sc1, int act,
                                bool emit_pre, int act_in, int flags) {
  Tensor a[8], b[8];
  bool keep[2] = {false, false};
  for (int i = 0; i < 8; ++i) {
    a[i] = opt(s0[i]);
    b[i] = opt(s1[i]);
    const bool ga = any_grad({&a[i]}), gb = any_grad({&b[i]});
    if (i != Stream::res && i != Stream::gate) {
      keep[0] |= ga;
      keep[1] |= gb;
    }
  }
  return FusedLinearPair::apply(wrap(a[0]), wrap(a[1]), wrap(a[2]), wrap(a[3]), wrap(a[4]), wrap(a[5]), wrap(a[6]), wrap(a[7]), wrap(b[0]), wrap(b[1]), wrap(b[2]), wrap(b[3]), wrap(b[4]), wrap(b[5]), wrap(b[6]), wrap(b[7]),
                                sc0, sc1, (int64_t)act, emit_pre, (int64_t)act_in, (int64_t)keep[0], (int64_t)keep[1],
                                (int64_t)flags);
}

// ------------------------------------------------------------------------------- linear + gated activation
// out[M, hidden] = glu(x W^T + b + s (x A^T) B^T) with W an up-projection [2 * hidden, K]: the gate is applied in
// the GEMM epilogue, so the [M, 2 * hidden] projection is written once for backward and never re-read in
// forward. The reference fuses the same pair in its feed-forward kernel
// (crates/training/src/sdxl/runtime.rs:249-321, host side :698-799).
namespace {

struct GluOut {
  Tensor y, x2, h, pre;
};
GluOut glu_forward(const Tensor& x, const Tensor& w, const Tensor& bias, const Tensor& la, const Tensor& lb, float s,
                   int code, bool keep, int flags) {
  GluOut r;
  r.x2 = contig(x).view({-1, x.size(-1)});
  const int64_t M = r.x2.size(0), N2 = w.size(0);
  GemmOpt o;
  if (keep) r.pre = empty_bf16({M, N2}, x);
  o.out = empty_bf16({M, N2 / 2}, x);
  if (la.defined()) r.h = skinny(r.x2, la, s, flags);
  o.bias = bias; o.lora_h = r.h; o.lora_b = lb; o.glu = code; o.pre_out = r.pre; o.pdl = flags & kPdl;
  auto shp = x.sizes().vec();
  shp.back() = N2 / 2;
  r.y = gemm(r.x2, w, o, flags).view(shp);
  return r;
}

struct FusedLinearGlu : torch::autograd::Function<FusedLinearGlu> {
  static Tensor forward(AutogradContext* ctx, const OptT& x_o, const OptT& w_o, const OptT& bias_o, const OptT& la_o,
                        const OptT& lb_o, const OptT& wt_o, double s, int64_t code, int64_t flags) {
    const Tensor x = opt(x_o), w = opt(w_o), bias = opt(bias_o), la = opt(la_o), lb = opt(lb_o), wt = opt(wt_o);
    if (ctx) ctx->saved_data["args"] = Args({&x, &w, &bias, &la, &lb, &wt}).mask;
    GluOut r = glu_forward(x, w, bias, la, lb, (float)s, (int)code, true, (int)flags);
    ctx->save_for_backward({r.x2, w, bias, la, lb, r.h, r.pre, wt});
    ctx->saved_data["s"] = s;
    ctx->saved_data["m"] = std::vector<int64_t>{code, flags};
    ctx->saved_data["shp"] = x.sizes().vec();
    return r.y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list gout) {
    auto sv = ctx->get_saved_variables();
    const auto m = ctx->saved_data["m"].toIntVector();
    const Tensor &x2 = sv[0], &w = sv[1], &bias = sv[2], &pre = sv[6];
    const int64_t M = x2.size(0), N2 = w.size(0);
    Tensor d2 = contig(gout[0]).view({M, N2 / 2});
    Tensor dh = empty_bf16({M, N2}, x2);
    const int code = (int)m[0];
    check(L.eri_glu_bwd(d2.data_ptr(), pre.data_ptr(), dh.data_ptr(), (int)M, (int)(N2 / 2), code == 1 || code == 3 ? 0 : 1,
                        code >= 3 ? 1 : 0, stream()), "glu_bwd");
    const Args args(ctx->saved_data["args"].toInt());
    auto need = [&](int i) { return args.need(ctx, i); };
    LinGrads g = linear_grads(dh, x2, w, bias, sv[3], sv[4], sv[5], (float)ctx->saved_data["s"].toDouble(), sv[7], need(0),
                              need(1), need(2), need(3), need(4), ctx->saved_data["shp"].toIntVector(),
                              (int)m[1]);
    return {g.dx, g.dw, g.db, g.da, g.dlb, Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

}  // namespace

Tensor linear_glu(const Tensor& x, const Tensor& w, const OptT& bias_, const OptT& la_, const OptT& lb_, double scale,
                  int code, const OptT& wt_, int flags) {
  Tensor bias = opt(bias_), la = opt(la_), lb = opt(lb_);
  if (any_grad({&x, &w, &bias, &la, &lb}))
    return FusedLinearGlu::apply(wrap(x), wrap(w), wrap(bias), wrap(la), wrap(lb), wt_, scale, (int64_t)code, (int64_t)flags);
  return glu_forward(x, w, bias, la, lb, (float)scale, code, false, flags).y;
}

// ----------------------------------------------------------------------------- conditioning-vector linear
// Linear on a handful of rows (T <= 8): bound by one pass over the weight in each direction.
Tensor small_wgrad(const Tensor& dy2, const Tensor& xin, double scale, const Tensor& accum) {
  const int64_t T = dy2.size(0), N = dy2.size(1), K = xin.size(1);
  Tensor dw = accum.defined() ? accum : empty_bf16({N, K}, dy2);
  check(L.eri_rows_wgrad(dy2.data_ptr(), (int)dy2.stride(0), xin.data_ptr(), (int)xin.stride(0), dw.data_ptr(), (int)K,
                         (int)T, (int)N, (int)K, accum.defined(), (float)scale, stream()), "rows_wgrad");
  return dw;
}

// dx[T, K] = dy2[T, N] w[N, K]; the fp32 partial planes are added in split order (deterministic).
Tensor small_dgrad(const Tensor& dy2, const Tensor& w) {
  const int64_t T = dy2.size(0), N = dy2.size(1), K = w.size(1);
  constexpr int kMaxSplits = 1024;
  Tensor part = empty_f32({kMaxSplits, T, K}, dy2);
  const int n = L.eri_rows_dgrad(dy2.data_ptr(), (int)dy2.stride(0), w.data_ptr(), (int)w.stride(0), (float*)part.data_ptr(),
                                 (int)T, (int)N, (int)K, kMaxSplits, stream());
  check(n > 0 ? 0 : (n ? n : -1), "rows_dgrad");
  return part.narrow(0, 0, n).sum(0).to(at::kBFloat16);
}

namespace {

Tensor small_forward(const Tensor& x, const Tensor& w, const Tensor& bias, bool silu_in, Tensor* x2_out) {
  Tensor x2 = contig(x).view({-1, x.size(-1)});
  const int64_t M = x2.size(0), K = x2.size(1), N = w.size(0);
  auto shp = x.sizes().vec();
  shp.back() = N;
  Tensor y = empty_bf16(shp, x);
  check(L.eri_gemv_bf16(x2.data_ptr(), w.data_ptr(), ptr(bias), y.data_ptr(), (int)M, (int)N, (int)K, (int)x2.stride(0),
                        (int)w.stride(0), (int)N, silu_in, 0, stream()), "gemv");
  if (x2_out) *x2_out = x2;
  return y;
}

struct SmallLinear : torch::autograd::Function<SmallLinear> {
  static Tensor forward(AutogradContext* ctx, const OptT& x_o, const OptT& w_o, const OptT& bias_o, bool silu_in, bool accum) {
    const Tensor x = opt(x_o), w = opt(w_o), bias = opt(bias_o);
    if (ctx) ctx->saved_data["args"] = Args({&x, &w, &bias}).mask;
    Tensor x2;
    Tensor y = small_forward(x, w, bias, silu_in, &x2);
    ctx->save_for_backward({x2, w, bias});
    ctx->saved_data["m"] = std::vector<int64_t>{silu_in, accum};
    ctx->saved_data["shp"] = x.sizes().vec();
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list gout) {
    auto sv = ctx->get_saved_variables();
    const Tensor &x2 = sv[0], &w = sv[1];
    const Args args(ctx->saved_data["args"].toInt());
    const auto m = ctx->saved_data["m"].toIntVector();
    const bool silu_in = m[0];
    const Tensor& dy = gout[0];
    Tensor dy2 = dy.reshape({-1, dy.size(-1)});
    if (dy2.stride(1) != 1) dy2 = dy2.contiguous();
    Tensor dx, dw, db;
    const bool native = x2.size(0) <= 8 && x2.size(1) % 8 == 0;
    if (args.need(ctx, 0)) {
      dx = native && rows_ok(w) ? small_dgrad(dy2, w) : at::mm(dy2, w);
      if (silu_in) dx = at::silu_backward(dx, x2);
      dx = dx.view(ctx->saved_data["shp"].toIntVector());
    }
    if (args.need(ctx, 1)) {
      Tensor xin = silu_in ? at::silu(x2) : x2;
      if (!native || !rows_ok(xin))
        dw = at::mm(dy2.t(), xin);
      else if (has_grad_buffer(w, at::kBFloat16, m[1]) && al16(w.grad()))
        small_wgrad(dy2, xin, 1.0, w.grad());      // added into the (arena) gradient view
      else
        dw = small_wgrad(dy2, xin, 1.0, Tensor());
    }
    if (args.need(ctx, 2)) db = dy2.sum(0);
    return {dx, dw, db, Tensor(), Tensor()};
  }
};

}  // namespace

Tensor small_linear(const Tensor& x, const Tensor& w, const OptT& bias_, bool silu_in, bool accum) {
  Tensor bias = opt(bias_);
  if (any_grad({&x, &w, &bias})) return SmallLinear::apply(wrap(x), wrap(w), wrap(bias), silu_in, accum);
  return small_forward(x, w, bias, silu_in, nullptr);
}

}  // namespace eri_ops
