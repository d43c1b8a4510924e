// Norms, QK-norm + rotary, gates, activations, attention, GroupNorm, losses and the fused single-stream block as
// autograd nodes over the kernels.
#include "eri_ops.h"

#include <ATen/cuda/CUDAGraphsUtils.cuh>

#include <map>
#include <mutex>

namespace eri_ops {

namespace {
Tensor to_bf16(const Tensor& t) { return t.defined() ? t.to(at::kBFloat16) : t; }
Tensor zeros_f32(at::IntArrayRef s, const Tensor& like) { return at::zeros(s, like.options().dtype(at::kFloat)); }
}  // namespace

// ------------------------------------------------------------------------------------- norm + modulation
namespace {

struct NormOut {
  Tensor y, x, scale, mean, rstd;
  int64_t stride;
};

NormOut norm_forward(const Tensor& x_, const Tensor& scale_, const Tensor& shift_, const Tensor& weight, const Tensor& bias,
                     double eps, bool rms) {
  NormOut r;
  r.x = contig(x_);
  const int64_t B = r.x.size(0), Lq = r.x.size(1), D = r.x.size(2);
  r.scale = mod_view(scale_, D);
  Tensor shift = mod_view(shift_, D);
  if (r.scale.defined() && shift.defined() && r.scale.stride(0) != shift.stride(0)) {
    r.scale = r.scale.contiguous();
    shift = shift.contiguous();
  }
  r.stride = r.scale.defined() ? r.scale.stride(0) : shift.defined() ? shift.stride(0) : D;
  r.y = at::empty_like(r.x);
  Tensor stats = empty_f32({2, B * Lq}, r.x);
  r.mean = stats.select(0, 0);
  r.rstd = stats.select(0, 1);
  int code = L.eri_norm_modulate_fwd_warp(r.x.data_ptr(), ptr(r.scale), ptr(shift), ptr(weight), ptr(bias), r.y.data_ptr(),
                                          (float*)r.mean.data_ptr(), (float*)r.rstd.data_ptr(), (int)(B * Lq), (int)D,
                                          (int)Lq, (int)r.stride, (float)eps, rms, stream());
  if (code == -100)
    code = L.eri_norm_modulate_fwd(r.x.data_ptr(), ptr(r.scale), ptr(shift), ptr(weight), ptr(bias), r.y.data_ptr(),
                                   (float*)r.mean.data_ptr(), (float*)r.rstd.data_ptr(), (int)(B * Lq), (int)D, (int)Lq,
                                   (int)r.stride, (float)eps, rms, stream());
  check(code, "norm_modulate_fwd");
  return r;
}

// ``skip``: also returns x itself for the residual branch around the norm; the gradient that comes back through it
// is added to dx inside the backward kernel instead of by a separate autograd sum.
struct NormModulate : torch::autograd::Function<NormModulate> {
  static variable_list forward(AutogradContext* ctx, const OptT& x_o, const OptT& scale_o, const OptT& shift_o,
                               const OptT& weight_o, const OptT& bias_o, double eps, bool rms, bool skip, bool accum) {
    const Tensor x = opt(x_o), scale = opt(scale_o), shift = opt(shift_o), weight = opt(weight_o), bias = opt(bias_o);
    if (ctx) ctx->saved_data["args"] = Args({&x, &scale, &shift, &weight, &bias}).mask;
    NormOut r = norm_forward(x, scale, shift, weight, bias, eps, rms);
    ctx->save_for_backward({r.x, r.scale, weight, bias, r.mean, r.rstd});
    ctx->saved_data["m"] = std::vector<int64_t>{r.stride, rms, skip, accum};
    ctx->set_materialize_grads(false);
    if (skip) return {r.y, r.x.view(r.x.sizes())};
    return {r.y};
  }
  static variable_list backward(AutogradContext* ctx, variable_list gout) {
    variable_list out(9);
    const auto m = ctx->saved_data["m"].toIntVector();
    Tensor dskip = m[2] ? gout[1] : Tensor();
    if (!gout[0].defined()) {       // the consumer had no gradient for this input (an unused stream)
      out[0] = dskip;
      return out;
    }
    auto sv = ctx->get_saved_variables();
    const Tensor &x = sv[0], &scale = sv[1], &weight = sv[2], &bias = sv[3], &mean = sv[4], &rstd = sv[5];
    const int64_t B = x.size(0), Lq = x.size(1), D = x.size(2), stride = m[0];
    const bool rms = m[1];
    Tensor dy = contig(gout[0]);
    const Args args(ctx->saved_data["args"].toInt());
    const bool want_sc = args.need(ctx, 1), want_sh = args.need(ctx, 2), want_w = args.need(ctx, 3), want_b = args.need(ctx, 4);
    const float *mu = (const float*)mean.data_ptr(), *rs = (const float*)rstd.data_ptr();
    Tensor dx = at::empty_like(x);
    bool added = false;
    // The gradients of scale and shift are column sums over a batch element's rows, those of weight and bias over
    // all rows: one column kernel next to the row kernel of dx. Scale together with trainable weight or bias mixes
    // the two and takes the general kernel.
    const bool mod = want_sc || want_sh, aff = want_w || want_b;
    const bool columns = !(mod && (weight.defined() || bias.defined())) && !(aff && scale.defined());
    int code = -100;
    if (columns) {
      Tensor dsk = dskip.defined() && dskip.scalar_type() == dx.scalar_type() ? contig(dskip) : Tensor();
      code = L.eri_norm_modulate_bwd_warp_add(dy.data_ptr(), x.data_ptr(), ptr(scale), ptr(weight), mu, rs, dx.data_ptr(),
                                              ptr(dsk), (int)(B * Lq), (int)D, (int)Lq, (int)stride, rms, stream());
      added = code != -100 && dsk.defined();
    }
    if (code != -100) {
      check(code, "norm_modulate_bwd");
      if (mod || aff) {
        Tensor d0, d1;      // sums of dy, of dy * xhat
        int acc = 0;
        if (mod) {
          if (want_sh) out[2] = d0 = empty_bf16({B, D}, x);
          if (want_sc) out[1] = d1 = empty_bf16({B, D}, x);
        } else {
          const bool acc_b = want_b && has_grad_buffer(bias, at::kBFloat16, m[3]), acc_w = want_w && has_grad_buffer(weight, at::kBFloat16, m[3]);
          if (want_b) d0 = acc_b ? bias.grad() : (out[4] = empty_bf16({D}, x));
          if (want_w) d1 = acc_w ? weight.grad() : (out[3] = empty_bf16({D}, x));
          acc = (acc_b ? 1 : 0) | (acc_w ? 2 : 0);
        }
        check(L.eri_col_norm_grad(dy.data_ptr(), x.data_ptr(), rms ? nullptr : mu, rs, mptr(d0), mptr(d1), mod ? (int)B : 1,
                                  (int)(mod ? Lq : B * Lq), (int)D, acc, stream()), "col_norm_grad");
      }
    } else {
      Tensor dsc = want_sc ? zeros_f32({B, D}, x) : Tensor(), dsh = want_sh ? zeros_f32({B, D}, x) : Tensor();
      Tensor dwt = want_w ? zeros_f32({D}, x) : Tensor(), dbs = want_b ? zeros_f32({D}, x) : Tensor();
      check(L.eri_norm_modulate_bwd(dy.data_ptr(), x.data_ptr(), ptr(scale), ptr(weight), ptr(bias), mu, rs, dx.data_ptr(),
                                    (float*)mptr(dsc), (float*)mptr(dsh), (float*)mptr(dwt), (float*)mptr(dbs), (int)(B * Lq),
                                    (int)D, (int)Lq, (int)stride, rms, stream()), "norm_modulate_bwd");
      out[1] = to_bf16(dsc); out[2] = to_bf16(dsh); out[3] = to_bf16(dwt); out[4] = to_bf16(dbs);
    }
    if (dskip.defined() && !added) dx = dx + dskip.view(dx.sizes());
    out[0] = dx;
    return out;
  }
};

}  // namespace

std::vector<Tensor> norm_modulate(const Tensor& x, const OptT& scale_, const OptT& shift_, const OptT& weight_,
                                  const OptT& bias_, double eps, bool rms, bool skip, bool accum) {
  Tensor scale = opt(scale_), shift = opt(shift_), weight = opt(weight_), bias = opt(bias_);
  if (any_grad({&x, &scale, &shift, &weight, &bias})) return NormModulate::apply(wrap(x), wrap(scale), wrap(shift), wrap(weight), wrap(bias), eps, rms, skip, accum);
  Tensor y = norm_forward(x, scale, shift, weight, bias, eps, rms).y;
  if (skip) return {y, x};
  return {y};
}

// --------------------------------------------------------------------------------------- QK-norm + RoPE
// Several token streams (e.g. text and image) -> one joint q, k, v of shape [B, sum(L_i), H, Dh]; each stream has
// its own QK-norm scales, the rotary table covers the joint sequence. One launch per stream writes straight into
// the joint tensors, so no concatenation copy exists in forward, and backward splits the gradient the same way.
namespace {

// [B, L, W] whose tokens may be row-strided (a column slice of a wider buffer)
Tensor tokmajor(const Tensor& t) {
  const bool ok = t.stride(2) == 1 && t.stride(0) == t.size(1) * t.stride(1) && t.stride(1) % 8 == 0 && al16(t);
  return ok ? t : t.contiguous();
}

void qknorm_fwd(const Tensor& qkv, int64_t tok_stride, const Tensor& qs, const Tensor& ks, const Tensor& cos, const Tensor& sin,
                Tensor& q, Tensor& k, Tensor& v, int64_t Li, int64_t off, double eps) {
  const int64_t B = q.size(0), Lt = q.size(1), H = q.size(2), Dh = q.size(3);
  check(L.eri_qknorm_rope_fwd(qkv.data_ptr(), ptr(qs), ptr(ks), (const float*)ptr(cos), (const float*)ptr(sin), q.data_ptr(),
                              k.data_ptr(), v.data_ptr(), (int)B, (int)Li, (int)H, (int)Dh, (int)Lt, (int)off, (float)eps,
                              (int)tok_stride, (int)(H * Dh), stream()), "qknorm_rope_fwd");
}

struct QKNormRope : torch::autograd::Function<QKNormRope> {
  // ``present``: the tensors of (qkv, q_scale, k_scale) per stream that exist, ``mask`` which those are
  static variable_list forward(AutogradContext* ctx, at::TensorList present, int64_t mask, int64_t n, const OptT& cos_o,
                               const OptT& sin_o, int64_t H, double eps) {
    const Tensor cos = opt(cos_o), sin = opt(sin_o);
    std::vector<Tensor> flat(3 * n);
    for (int64_t i = 0, k = 0; i < 3 * n; ++i)
      if ((mask >> i) & 1) flat[i] = present[k++];
    const int64_t B = flat[0].size(0), W = flat[0].size(2), Dh = W / (3 * H);
    int64_t Lt = 0;
    for (int64_t i = 0; i < n; ++i) Lt += flat[3 * i].size(1);
    Tensor q = empty_bf16({B, Lt, H, Dh}, flat[0]), k = at::empty_like(q), v = at::empty_like(q);
    variable_list save{cos, sin};
    int64_t off = 0;
    for (int64_t i = 0; i < n; ++i) {
      Tensor t = tokmajor(flat[3 * i]);
      qknorm_fwd(t, t.stride(1), flat[3 * i + 1], flat[3 * i + 2], cos, sin, q, k, v, t.size(1), off, eps);
      off += t.size(1);
      save.push_back(t);
      save.push_back(flat[3 * i + 1]);
      save.push_back(flat[3 * i + 2]);
    }
    ctx->save_for_backward(save);
    ctx->saved_data["m"] = std::vector<int64_t>{n, H, Lt, mask};
    ctx->saved_data["eps"] = eps;
    return {q, k, v};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto sv = ctx->get_saved_variables();
    const auto m = ctx->saved_data["m"].toIntVector();
    const int64_t n = m[0], H = m[1], Lt = m[2];
    Tensor dq = contig(g[0]), dk = contig(g[1]), dv = contig(g[2]);
    const int64_t B = dq.size(0), Dh = dq.size(3);
    const Args args(m[3]);
    const int64_t n_present = __builtin_popcountll((uint64_t)m[3]);
    variable_list out(n_present + 6);
    int64_t off = 0, slot = 0;
    for (int64_t i = 0; i < n; ++i) {
      const Tensor &qkv = sv[2 + 3 * i], &qs = sv[3 + 3 * i], &ks = sv[4 + 3 * i];
      Tensor d = at::empty(qkv.sizes(), qkv.options());
      const bool nq = args.need(ctx, (int)(3 * i + 1)), nk = args.need(ctx, (int)(3 * i + 2));
      Tensor dqs = nq ? zeros_f32({Dh}, dq) : Tensor(), dks = nk ? zeros_f32({Dh}, dq) : Tensor();
      check(L.eri_qknorm_rope_bwd(dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), qkv.data_ptr(), ptr(qs), ptr(ks),
                                  (const float*)ptr(sv[0]), (const float*)ptr(sv[1]), d.data_ptr(), (float*)mptr(dqs),
                                  (float*)mptr(dks), (int)B, (int)qkv.size(1), (int)H, (int)Dh, (int)Lt, (int)off,
                                  (float)ctx->saved_data["eps"].toDouble(), (int)qkv.stride(1), (int)(H * Dh), (int)d.stride(1),
                                  stream()), "qknorm_rope_bwd");
      off += qkv.size(1);
      out[slot++] = d;
      if (qs.defined()) out[slot++] = to_bf16(dqs);
      if (ks.defined()) out[slot++] = to_bf16(dks);
    }
    return out;
  }
};

}  // namespace

std::vector<Tensor> qknorm_rope_joint(const std::vector<OptT>& flat, const OptT& cos, const OptT& sin, int64_t heads,
                                      double eps) {
  std::vector<Tensor> f;
  bool grad = false;
  const Tensor cos_t = opt(cos), sin_t = opt(sin);
  refuse_tangents({&cos_t, &sin_t});
  for (auto& t : flat) {
    f.push_back(opt(t));
    grad |= any_grad({&f.back()});
  }
  if (grad) {
    std::vector<Tensor> present;
    int64_t mask = 0;
    for (size_t i = 0; i < f.size(); ++i)
      if (f[i].defined()) {
        mask |= 1ll << i;
        present.push_back(f[i]);
      }
    return QKNormRope::apply(at::TensorList(present), mask, (int64_t)f.size() / 3, cos, sin, heads, eps);
  }
  const int64_t B = f[0].size(0), Dh = f[0].size(2) / (3 * heads);
  int64_t Lt = 0, off = 0;
  for (size_t i = 0; i < f.size(); i += 3) Lt += f[i].size(1);
  Tensor q = empty_bf16({B, Lt, heads, Dh}, f[0]), k = at::empty_like(q), v = at::empty_like(q);
  for (size_t i = 0; i < f.size(); i += 3) {
    Tensor t = tokmajor(f[i]);
    qknorm_fwd(t, t.stride(1), f[i + 1], f[i + 2], opt(cos), opt(sin), q, k, v, t.size(1), off, eps);
    off += t.size(1);
  }
  return {q, k, v};
}

// --------------------------------------------------------------------------------------- gate + residual
namespace {

Tensor gate_forward(const Tensor& x, const Tensor& y, const Tensor& gate_v) {
  const int64_t D = y.size(2), Lq = y.size(1);
  Tensor out = at::empty_like(y);
  check(L.eri_gate_residual(ptr(x), y.data_ptr(), ptr(gate_v), out.data_ptr(), y.numel() / D, (int)D, (int)Lq,
                            gate_v.defined() ? (int)gate_v.stride(0) : 0, stream()), "gate_residual");
  return out;
}

struct GateResidual : torch::autograd::Function<GateResidual> {
  static Tensor forward(AutogradContext* ctx, const OptT& x_o, const OptT& y_in_o, const OptT& gate_o, bool keep_y) {
    const Tensor x = opt(x_o), y_in = opt(y_in_o), gate = opt(gate_o);
    if (ctx) ctx->saved_data["args"] = Args({&x, &y_in, &gate}).mask;
    Tensor y = contig(y_in), gate_v = mod_view(gate, y.size(2));
    ctx->save_for_backward({keep_y ? y : Tensor(), gate_v});
    ctx->saved_data["m"] = std::vector<int64_t>{x.defined(), y.size(0), y.size(1), y.size(2)};
    return gate_forward(contig(x), y, gate_v);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto sv = ctx->get_saved_variables();
    const auto m = ctx->saved_data["m"].toIntVector();
    Tensor dout = contig(g[0]), dx = m[0] ? dout : Tensor();
    if (!sv[1].defined()) return {dx, dout, Tensor(), Tensor()};
    Tensor dy = gate_forward(Tensor(), dout, sv[1]), dg;
    if (Args(ctx->saved_data["args"].toInt()).need(ctx, 2)) {
      dg = empty_bf16({m[1], m[3]}, dout);
      check(L.eri_col_dot(dout.data_ptr(), sv[0].data_ptr(), dg.data_ptr(), (int)m[1], (int)m[2], (int)m[3], stream()), "col_dot");
    }
    return {dx, dy, dg, Tensor()};
  }
};

}  // namespace

Tensor gate_residual(const OptT& x_, const Tensor& y, const OptT& gate_) {
  Tensor x = opt(x_), gate = opt(gate_);
  if (any_grad({&x, &y, &gate})) return GateResidual::apply(wrap(x), wrap(y), wrap(gate), gate.defined() && gate.requires_grad());
  Tensor yc = contig(y);
  return gate_forward(contig(x), yc, mod_view(gate, y.size(2)));
}

// (x[:, :n], x[:, n:]) as views. Autograd's own slice backward allocates a zero tensor of x's size per slice, copies
// the slice's gradient into it and sums the two; here the backward is one concatenation.
namespace {
struct SplitTokens : torch::autograd::Function<SplitTokens> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, int64_t n) {
    ctx->saved_data["n"] = n;
    ctx->saved_data["shp"] = x.sizes().vec();
    ctx->set_materialize_grads(false);
    return {x.narrow(1, 0, n), x.narrow(1, n, x.size(1) - n)};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    if (!g[0].defined() && !g[1].defined()) return {Tensor(), Tensor()};
    auto shp = ctx->saved_data["shp"].toIntVector();
    const int64_t n = ctx->saved_data["n"].toInt(), total = shp[1];
    for (int i = 0; i < 2; ++i)
      if (!g[i].defined()) {
        shp[1] = i ? total - n : n;
        g[i] = at::zeros(shp, g[1 - i].options());
      }
    return {at::cat({g[0], g[1]}, 1), Tensor()};
  }
};
}  // namespace
std::vector<Tensor> split_tokens(const Tensor& x, int64_t n) {
  if (any_grad({&x})) return SplitTokens::apply(x, n);
  return {x.narrow(1, 0, n), x.narrow(1, n, x.size(1) - n)};
}

// --------------------------------------------------------------------------------------- activations, GLU
namespace {
struct Act : torch::autograd::Function<Act> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x_, int64_t mode) {
    Tensor x = contig(x_), y = at::empty_like(x);
    check(L.eri_act_fwd(x.data_ptr(), y.data_ptr(), x.numel(), (int)mode, stream()), "act_fwd");
    ctx->save_for_backward({x});
    ctx->saved_data["m"] = mode;
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    Tensor x = ctx->get_saved_variables()[0], dy = contig(g[0]), dx = at::empty_like(x);
    check(L.eri_act_bwd(dy.data_ptr(), x.data_ptr(), dx.data_ptr(), x.numel(), (int)ctx->saved_data["m"].toInt(), stream()),
          "act_bwd");
    return {dx, Tensor()};
  }
};

Tensor glu_fwd(const Tensor& h, int64_t mode, bool act_first) {
  const int64_t F2 = h.size(-1);
  auto shp = h.sizes().vec();
  shp.back() = F2 / 2;
  Tensor out = empty_bf16(shp, h);
  check(L.eri_glu_fwd(h.data_ptr(), out.data_ptr(), (int)(h.numel() / F2), (int)(F2 / 2), (int)mode, act_first, stream()),
        "glu_fwd");
  return out;
}
struct Glu : torch::autograd::Function<Glu> {
  static Tensor forward(AutogradContext* ctx, const Tensor& h_, int64_t mode, bool act_first) {
    Tensor h = contig(h_);
    ctx->save_for_backward({h});
    ctx->saved_data["m"] = std::vector<int64_t>{mode, act_first};
    return glu_fwd(h, mode, act_first);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    Tensor h = ctx->get_saved_variables()[0], dout = contig(g[0]), dh = at::empty_like(h);
    const auto m = ctx->saved_data["m"].toIntVector();
    const int64_t F2 = h.size(-1);
    check(L.eri_glu_bwd(dout.data_ptr(), h.data_ptr(), dh.data_ptr(), (int)(h.numel() / F2), (int)(F2 / 2), (int)m[0], (int)m[1],
                        stream()), "glu_bwd");
    return {dh, Tensor(), Tensor()};
  }
};
}  // namespace

Tensor act(const Tensor& x, int mode) {
  if (any_grad({&x})) return Act::apply(x, (int64_t)mode);
  Tensor xc = contig(x), y = at::empty_like(xc);
  check(L.eri_act_fwd(xc.data_ptr(), y.data_ptr(), xc.numel(), mode, stream()), "act_fwd");
  return y;
}
Tensor glu(const Tensor& h, int mode, bool act_first) {
  if (any_grad({&h})) return Glu::apply(h, (int64_t)mode, act_first);
  return glu_fwd(contig(h), mode, act_first);
}

// ----------------------------------------------------------------------------------------------- attention
namespace {

// Key bias (log2 units) that blanks the padding of a key set shorter than one tile: [B, 128] rows followed by one
// flag per (batch, tile), all set. Constant per (B, Lk, device): the first kMaxPad shapes are made once and kept for
// good (any stream may be reading one, so none is ever given back); later shapes, and shapes first met while a graph
// is captured, are made by the call on its own stream (three small launches).
Tensor make_pad_bias(int64_t B, int64_t Lk, const Tensor& like) {
  Tensor t = at::full({B * 128 + B}, -1.0e30f, like.options().dtype(at::kFloat));
  t.narrow(0, 0, B * 128).view({B, 128}).narrow(1, 0, Lk).zero_();
  t.narrow(0, B * 128, B).view(at::kInt).fill_(1);
  return t;
}
Tensor pad_bias(int64_t B, int64_t Lk, const Tensor& like) {
  constexpr size_t kMaxPad = 64;
  static std::mutex mu;
  static std::map<std::tuple<int64_t, int64_t, int>, Tensor> cache;
  const auto key = std::make_tuple(B, Lk, (int)like.device().index());
  std::lock_guard<std::mutex> lock(mu);
  auto it = cache.find(key);
  if (it != cache.end()) return it->second;
  Tensor t = make_pad_bias(B, Lk, like);
  if (cache.size() < kMaxPad && at::cuda::currentStreamCaptureStatus() == at::cuda::CaptureStatus::None) {
    c10::cuda::getCurrentCUDAStream().synchronize();      // another stream may read it from now on
    cache[key] = t;
  }
  return t;
}

}  // namespace

namespace {

// Token stride of a [B, L, H, D] operand the kernels read or write in place (heads packed), 0 where there is none. The
// stride of a dimension of size 1 says nothing: a contiguous tensor may have any value there.
int64_t token_stride(const Tensor& t) {
  const int64_t B = t.size(0), L_ = t.size(1), H = t.size(2), D = t.size(3);
  const int64_t ld = L_ > 1 ? t.stride(1) : B > 1 ? t.stride(0) : H * D;
  const bool ok = t.stride(3) == 1 && (H == 1 || t.stride(2) == D) && ld >= H * D && ld % 8 == 0 && al16(t) &&
                  (B == 1 || t.stride(0) == L_ * ld);
  return ok ? ld : 0;
}
Tensor packed_heads(const Tensor& t) { return token_stride(t) ? t : contig16(t); }

}  // namespace

std::pair<Tensor, Tensor> attn_fwd(const Tensor& q, const Tensor& k, const Tensor& v, double scale, const Tensor& out_,
                                   const Tensor& kbias, int pair_poly) {
  const int64_t B = q.size(0), Lq = q.size(1), H = q.size(2), D = q.size(3), Lk = k.size(1);
  Tensor out = out_.defined() ? out_ : empty_bf16({B, Lq, H, D}, q);
  EriAttnStrides ld = {};
  ld.q = token_stride(q); ld.k = token_stride(k); ld.v = token_stride(v); ld.out = token_stride(out);
  TORCH_CHECK_VALUE(ld.q && ld.k && ld.v && ld.out, "flash attention: unsupported operand strides");
  // the kernels walk the keys with q's batch, head count and head size
  TORCH_CHECK_VALUE(k.size(0) == B && k.size(2) == H && k.size(3) == D && v.sizes() == k.sizes(), "flash attention: q ", q.sizes(),
                    " does not go with k ", k.sizes(), " and v ", v.sizes());
  Tensor lse = empty_f32({B, H, Lq}, q);
  if (pair_poly >= 0 && !kbias.defined() && out.is_contiguous() && q.is_contiguous() && k.is_contiguous() &&
      v.is_contiguous() && D == 128 && Lq >= 256 && Lk >= 128) {
    const int code = L.eri_flash_attn_fwd_pair(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), (float*)lse.data_ptr(),
                                               (int)B, (int)H, (int)Lq, (int)Lk, (int)D, (float)scale, pair_poly, stream());
    if (code != -100) return check(code, "flash_attn_fwd_pair"), std::pair<Tensor, Tensor>{out, lse};
  }
  check(L.eri_flash_attn_fwd_strided(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), (float*)lse.data_ptr(),
                                     (const float*)ptr(kbias), (int)B, (int)H, (int)Lq, (int)Lk, (int)D, (float)scale, &ld,
                                     stream()), "flash_attn_fwd");
  return {out, lse};
}

// dq, dk, dv: where the gradients go (heads packed, any token stride).
void attn_bwd_into(const Tensor& dout, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& out, const Tensor& lse,
                   double scale, const Tensor& kbias, const Tensor& dq, const Tensor& dk, const Tensor& dv) {
  const int64_t B = q.size(0), Lq = q.size(1), H = q.size(2), D = q.size(3), Lk = k.size(1), Lp = (Lq + 127) / 128 * 128;
  Tensor aux = empty_f32({2, B, H, Lp}, q);
  float *lse2 = (float*)aux.data_ptr(), *delta = lse2 + B * H * Lp;
  EriAttnStrides ld = {};
  ld.q = token_stride(q); ld.k = token_stride(k); ld.v = token_stride(v); ld.out = token_stride(out);
  ld.dq = token_stride(dq); ld.dk = token_stride(dk); ld.dv = token_stride(dv);
  check(L.eri_flash_attn_bwd_strided(dout.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(),
                                     (const float*)lse.data_ptr(), lse2, delta, dq.data_ptr(), dk.data_ptr(), dv.data_ptr(),
                                     (const float*)ptr(kbias), (int)B, (int)H, (int)Lq, (int)Lk, (int)D, (float)scale, &ld,
                                     stream()), "flash_attn_bwd");
}

std::tuple<Tensor, Tensor, Tensor> attn_bwd(const Tensor& dout, const Tensor& q, const Tensor& k, const Tensor& v,
                                            const Tensor& out, const Tensor& lse, double scale, const Tensor& kbias) {
  Tensor dq = empty_bf16(q.sizes(), q), dk = empty_bf16(k.sizes(), k), dv = empty_bf16(v.sizes(), v);
  attn_bwd_into(dout, q, k, v, out, lse, scale, kbias, dq, dk, dv);
  return {dq, dk, dv};
}

namespace {

struct Attention : torch::autograd::Function<Attention> {
  static Tensor forward(AutogradContext* ctx, const OptT& q_o, const OptT& k_o, const OptT& v_o, const OptT& kbias_o, double scale,
                        int64_t pair_poly) {
    const Tensor q = packed_heads(*q_o), k = packed_heads(*k_o), v = packed_heads(*v_o), kbias = opt(kbias_o);
    auto [out, lse] = attn_fwd(q, k, v, scale, Tensor(), kbias, (int)pair_poly);
    ctx->save_for_backward({q, k, v, out, lse, kbias});
    ctx->saved_data["s"] = scale;
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto sv = ctx->get_saved_variables();
    auto [dq, dk, dv] = attn_bwd(contig16(g[0]), sv[0], sv[1], sv[2], sv[3], sv[4], ctx->saved_data["s"].toDouble(), sv[5]);
    return {dq, dk, dv, Tensor(), Tensor(), Tensor()};
  }
};

// Attention whose operands are column blocks of projections' outputs, read in place; the gradients are written as the
// column blocks of the projections' output gradients. ``kv`` undefined: q, k and v are all in ``a`` [B, L, 3 * H * D]
// (self-attention); else a = q [B, L, H * D] and kv [B, Lk, 2 * H * D]. Neither direction has a split, concatenation
// or copy of its own.
struct Parts {
  Tensor q, k, v;
  Parts(const Tensor& a, const Tensor& kv, int64_t H) {
    const int64_t B = a.size(0), Lq = a.size(1);
    if (kv.defined()) {
      const int64_t D = a.size(2) / H;
      Tensor s = kv.view({B, kv.size(1), 2, H, D});
      q = a.view({B, Lq, H, D});
      k = s.select(2, 0);
      v = s.select(2, 1);
    } else {
      Tensor s = a.view({B, Lq, 3, H, a.size(2) / (3 * H)});
      q = s.select(2, 0);
      k = s.select(2, 1);
      v = s.select(2, 2);
    }
  }
};
struct PackedAttention : torch::autograd::Function<PackedAttention> {
  static Tensor forward(AutogradContext* ctx, const OptT& a_o, const OptT& kv_o, const OptT& kbias_o, int64_t heads, double scale) {
    const Tensor a = contig16(opt(a_o)), kv = contig16(opt(kv_o)), kbias = opt(kbias_o);
    Parts p(a, kv, heads);
    auto [out, lse] = attn_fwd(p.q, p.k, p.v, scale, Tensor(), kbias, -1);
    ctx->save_for_backward({a, kv, out, lse, kbias});
    ctx->saved_data["s"] = scale;
    ctx->saved_data["h"] = heads;
    return out.flatten(2);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto sv = ctx->get_saved_variables();
    const int64_t heads = ctx->saved_data["h"].toInt();
    Tensor da = empty_bf16(sv[0].sizes(), sv[0]), dkv;
    if (sv[1].defined()) dkv = empty_bf16(sv[1].sizes(), sv[1]);
    Parts p(sv[0], sv[1], heads), d(da, dkv, heads);
    attn_bwd_into(contig16(g[0]), p.q, p.k, p.v, sv[2], sv[3], ctx->saved_data["s"].toDouble(), sv[4], d.q, d.k, d.v);
    return {da, dkv, Tensor(), Tensor(), Tensor()};
  }
};

Tensor packed_attention(const Tensor& a, const Tensor& kv, int64_t heads, double scale, const OptT& kbias_) {
  Tensor kbias = opt(kbias_);
  const int64_t Lk = kv.defined() ? kv.size(1) : a.size(1);
  if (!kbias.defined() && Lk < 128) kbias = pad_bias(a.size(0), Lk, a);
  refuse_tangents({&kbias});
  if (any_grad({&a, &kv})) return PackedAttention::apply(wrap(a), wrap(kv), wrap(kbias), heads, scale);
  Parts p(contig16(a), contig16(kv), heads);
  return attn_fwd(p.q, p.k, p.v, scale, Tensor(), kbias, -1).first.flatten(2);
}

}  // namespace

// q, k, v [B, L, H, Dh]; kbias from flash_attn.key_bias or none. pair_poly < 0: one-CTA forward.
Tensor attention(const Tensor& q, const Tensor& k, const Tensor& v, double scale, const OptT& kbias_, int pair_poly) {
  Tensor kbias = opt(kbias_);
  if (!kbias.defined() && k.size(1) < 128) kbias = pad_bias(k.size(0), k.size(1), q);
  refuse_tangents({&kbias});
  if (any_grad({&q, &k, &v})) return Attention::apply(wrap(q), wrap(k), wrap(v), wrap(kbias), scale, (int64_t)pair_poly);
  return attn_fwd(packed_heads(q), packed_heads(k), packed_heads(v), scale, Tensor(), kbias, pair_poly).first;
}
Tensor attention_qkv(const Tensor& qkv, int64_t heads, double scale, const OptT& kbias) {
  return packed_attention(qkv, Tensor(), heads, scale, kbias);
}
Tensor attention_kv(const Tensor& q, const Tensor& kv, int64_t heads, double scale, const OptT& kbias) {
  return packed_attention(q, kv, heads, scale, kbias);
}

// q, k, v [B, L, H, 512] (column blocks of wider tensors are read in place), no gradient.
Tensor attention_wide(const Tensor& q_, const Tensor& k_, const Tensor& v_, double scale) {
  refuse_tangents({&q_, &k_, &v_});
  const Tensor q = packed_heads(q_), k = packed_heads(k_), v = packed_heads(v_);
  const int64_t B = q.size(0), Lq = q.size(1), H = q.size(2), Lk = k.size(1);
  TORCH_CHECK_VALUE(q.size(3) == 512 && k.sizes() == v.sizes() && k.size(0) == B && k.size(2) == H && k.size(3) == 512,
                    "attention_wide: operand sizes");
  Tensor out = empty_bf16({B, Lq, H, 512}, q);
  EriAttnStrides ld = {};
  ld.q = token_stride(q); ld.k = token_stride(k); ld.v = token_stride(v);
  TORCH_CHECK_VALUE(ld.q && ld.k && ld.v, "attention_wide: unsupported operand strides");
  check(L.eri_flash_attn_wide_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), (int)B, (int)H, (int)Lq, (int)Lk,
                                  (float)scale, &ld, stream()), "flash_attn_wide");
  return out;
}

// q, k, v [B, L, H, 64 | 128] (column blocks of wider tensors are read in place) with an additive bf16 or boolean mask
// that broadcasts to [B, H, Lq, Lk]; no gradient.
Tensor attention_bias(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& bias, double scale) {
  refuse_tangents({&q_, &k_, &v_, &bias});
  const Tensor q = packed_heads(q_), k = packed_heads(k_), v = packed_heads(v_);
  const int64_t B = q.size(0), Lq = q.size(1), H = q.size(2), D = q.size(3), Lk = k.size(1);
  const bool is_bool = bias.scalar_type() == at::kBool;
  TORCH_CHECK_VALUE(k.sizes() == v.sizes() && k.size(0) == B && k.size(2) == H && k.size(3) == D && bias.device() == q.device() &&
                        (is_bool || bias.scalar_type() == at::kBFloat16) && bias.dim() == 4 && bias.size(3) == Lk,
                    "attention_bias: operands");
  Tensor m = (bias.stride(3) == 1 || Lk == 1 ? bias : bias.contiguous()).expand({B, H, Lq, Lk});
  Tensor out = empty_bf16({B, Lq, H, D}, q);
  EriAttnStrides ld = {};
  ld.q = token_stride(q); ld.k = token_stride(k); ld.v = token_stride(v);
  TORCH_CHECK_VALUE(ld.q && ld.k && ld.v, "attention_bias: unsupported operand strides");
  check(L.eri_flash_attn_bias_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), m.data_ptr(), m.stride(0), m.stride(1),
                                  m.stride(2), is_bool, (int)B, (int)H, (int)Lq, (int)Lk, (int)D, (float)scale, &ld, stream()),
        "flash_attn_bias");
  return out;
}

// Self-attention of a packed projection whose queries and keys are first normalised (RMS over the whole width) and
// rotated: attention(rope(norm(q) * wq), rope(norm(k) * wk), v). q, k, v are read and their gradients written inside
// the packed tensors.
namespace {

// fp32 table the kernels can read in 16-byte words
Tensor rope_rows(const Tensor& t) {
  Tensor f = t.to(at::kFloat);
  return f.stride(1) == 1 && f.stride(0) % 4 == 0 && al16(f) ? f : contig16(f);
}

struct RopeAttention : torch::autograd::Function<RopeAttention> {
  static Tensor forward(AutogradContext* ctx, const OptT& qkv_o, const OptT& wq_o, const OptT& wk_o, const OptT& cos_o,
                        const OptT& sin_o, int64_t heads, double eps, bool keep) {
    const Tensor qkv = contig16(*qkv_o), wq = contig16(*wq_o), wk = contig16(*wk_o);
    const int64_t B = qkv.size(0), Lq = qkv.size(1), D = qkv.size(2) / 3;
    Tensor cos = rope_rows(*cos_o), sin = rope_rows(*sin_o);
    if (cos.stride(0) != sin.stride(0)) {
      cos = contig16(cos);
      sin = contig16(sin);
    }
    Parts p(qkv, Tensor(), heads);
    Tensor q = empty_bf16({B, Lq, heads, D / heads}, qkv), k = at::empty_like(q), rstd = empty_f32({2, B * Lq}, qkv);
    check(L.eri_norm_rope_fwd(p.q.data_ptr(), p.k.data_ptr(), 3 * D, wq.data_ptr(), wk.data_ptr(), (const float*)cos.data_ptr(),
                              (const float*)sin.data_ptr(), cos.stride(0), q.data_ptr(), k.data_ptr(), (float*)rstd.data_ptr(),
                              (int)(B * Lq), (int)Lq, (int)D, (float)eps, stream()), "norm_rope_fwd");
    Tensor kbias = Lq < 128 ? pad_bias(B, Lq, qkv) : Tensor();
    auto [out, lse] = attn_fwd(q, k, p.v, 1.0 / std::sqrt((double)(D / heads)), Tensor(), kbias, -1);
    if (keep) {
      ctx->save_for_backward({qkv, wq, wk, cos, sin, rstd, q, k, out, lse, kbias});
      ctx->saved_data["h"] = heads;
    }
    return out.flatten(2);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto sv = ctx->get_saved_variables();
    const Tensor &qkv = sv[0], &wq = sv[1], &wk = sv[2], &cos = sv[3], &sin = sv[4], &rstd = sv[5], &q = sv[6], &k = sv[7];
    const int64_t heads = ctx->saved_data["h"].toInt(), B = q.size(0), Lq = q.size(1), D = q.size(2) * q.size(3);
    Tensor d_qkv = empty_bf16(qkv.sizes(), qkv), dq = at::empty_like(q), dk = at::empty_like(k);
    Parts p(qkv, Tensor(), heads), d(d_qkv, Tensor(), heads);
    attn_bwd_into(contig16(g[0]), q, k, p.v, sv[8], sv[9], 1.0 / std::sqrt((double)(D / heads)), sv[10], dq, dk, d.v);
    check(L.eri_norm_rope_bwd(p.q.data_ptr(), p.k.data_ptr(), 3 * D, wq.data_ptr(), wk.data_ptr(), (const float*)cos.data_ptr(),
                              (const float*)sin.data_ptr(), cos.stride(0), (const float*)rstd.data_ptr(), dq.data_ptr(),
                              dk.data_ptr(), d.q.data_ptr(), d.k.data_ptr(), 3 * D, (int)(B * Lq), (int)Lq, (int)D, stream()),
          "norm_rope_bwd");
    return {d_qkv, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

}  // namespace

// wq, wk [D] and the tables [L, D / 2] get no gradient (the caller keeps to the separate ops where they need one).
Tensor attention_qkv_rope(const Tensor& qkv, const Tensor& wq, const Tensor& wk, const Tensor& cos, const Tensor& sin,
                          int64_t heads, double eps) {
  const int64_t D = qkv.size(2) / 3;
  TORCH_CHECK_VALUE(wq.numel() == D && wk.numel() == D && cos.dim() == 2 && cos.size(0) == qkv.size(1) && cos.size(1) * 2 == D &&
                        sin.sizes() == cos.sizes(), "attention_qkv_rope: operand sizes");
  refuse_tangents({&wq, &wk, &cos, &sin});
  if (any_grad({&qkv})) return RopeAttention::apply(wrap(qkv), wrap(wq), wrap(wk), wrap(cos), wrap(sin), heads, eps, true);
  return RopeAttention::forward(nullptr, qkv, wq, wk, cos, sin, heads, eps, false);
}

// ---------------------------------------------------------------------------------------------------- loss
namespace {
struct MseLoss : torch::autograd::Function<MseLoss> {
  static Tensor forward(AutogradContext* ctx, const OptT& pred__o, const OptT& target__o, const OptT& weight_o) {
    const Tensor pred_ = opt(pred__o), target_ = opt(target__o), weight = opt(weight_o);
    if (ctx) ctx->saved_data["args"] = Args({&pred_, &target_, &weight}).mask;
    Tensor pred = contig(pred_), target = contig(target_);
    const int64_t n = pred.numel();
    Tensor loss = zeros_f32({}, pred), dpred = at::empty_like(pred);
    Tensor w = weight.defined() ? weight.to(at::kFloat).contiguous() : weight;
    check(L.eri_mse_fwd_bwd(pred.data_ptr(), target.data_ptr(), (const float*)ptr(w), (float*)loss.data_ptr(), dpred.data_ptr(), n,
                            n / pred.size(0), 1.f, stream()), "mse");
    ctx->save_for_backward({dpred});
    return loss;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    Tensor dpred = ctx->get_saved_variables()[0];
    return {dpred * g[0].to(dpred.scalar_type()), Tensor(), Tensor()};
  }
};
}  // namespace
Tensor mse_loss(const Tensor& pred, const Tensor& target, const OptT& weight) {
  const Tensor w = opt(weight);
  refuse_tangents({&pred, &target, &w});
  return MseLoss::apply(wrap(pred), wrap(target), weight);
}

// ------------------------------------------------------------------------ channels-last convolution helpers
// Activations are [N, HW, C] rows or [N, C, H, W] in channels-last format (the same memory); results keep the form.
namespace {

struct Rows {
  int N, HW, C;
  explicit Rows(const Tensor& x) {
    N = (int)x.size(0);
    C = (int)(x.dim() == 4 ? x.size(1) : x.size(2));
    HW = (int)(x.dim() == 4 ? x.size(2) * x.size(3) : x.size(1));
  }
};
Tensor rows_contig(const Tensor& x) {
  Tensor c = x.dim() == 4 ? x.contiguous(at::MemoryFormat::ChannelsLast) : contig(x);
  return al16(c) ? c : c.clone();      // (a clone keeps the memory format)
}

// The kernels index these by channel (and sample): a shorter tensor would be read past its end.
void check_channels(const Tensor& t, int64_t n, const char* what) {
  TORCH_CHECK_VALUE(!t.defined() || t.numel() == n, what, ": ", t.sizes(), " where ", n, " values are needed");
}

// GroupNorm (+SiLU) of x + pre_c + pre_nc: the bias of the convolution before it and a per-sample embedding are added
// where x is read.
Tensor gn_forward(const Tensor& x, const Tensor& w, const Tensor& b, const Tensor& pc, const Tensor& pn, int64_t groups,
                  double eps, bool silu, const Tensor& stats) {
  const Rows r(x);
  Tensor y = at::empty_like(x), ws = empty_f32({L.eri_gn_workspace(r.N, r.HW, r.C, (int)groups, 0)}, x);
  float* st = stats.defined() ? (float*)stats.data_ptr() : nullptr;
  check(L.eri_gn_fwd(x.data_ptr(), ptr(pc), ptr(pn), w.data_ptr(), ptr(b), y.data_ptr(), st, st ? st + r.N * groups : nullptr,
                     (float*)ws.data_ptr(), r.N, r.HW, r.C, (int)groups, (float)eps, silu, stream()), "gn_fwd");
  return y;
}
struct GroupNormSilu : torch::autograd::Function<GroupNormSilu> {
  static Tensor forward(AutogradContext* ctx, const OptT& x_o, const OptT& w_o, const OptT& b_o, const OptT& pc_o,
                        const OptT& pn_o, int64_t groups, double eps, bool silu, bool accum) {
    const Tensor x = rows_contig(*x_o), w = contig16(*w_o), b = contig16(opt(b_o)), pc = contig16(opt(pc_o)), pn = contig16(opt(pn_o));
    ctx->saved_data["args"] = Args({&x, &w, &b, &pc, &pn}).mask;
    Tensor stats = empty_f32({2, x.size(0), groups}, x);
    Tensor y = gn_forward(x, w, b, pc, pn, groups, eps, silu, stats);
    ctx->save_for_backward({x, w, b, stats, pc, pn});
    ctx->saved_data["m"] = std::vector<int64_t>{groups, silu, accum};
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto sv = ctx->get_saved_variables();
    const Tensor &x = sv[0], &w = sv[1], &b = sv[2], &stats = sv[3], &pc = sv[4], &pn = sv[5];
    const auto m = ctx->saved_data["m"].toIntVector();
    const int G = (int)m[0];
    const Rows r(x);
    Tensor dy = rows_contig(g[0]), dx = at::empty_like(x), ws = empty_f32({L.eri_gn_workspace(r.N, r.HW, r.C, G, 1)}, x);
    const Args args(ctx->saved_data["args"].toInt());
    // a parameter's gradient goes straight into its buffer when it has one
    variable_list out(9);
    int acc = 0;
    auto dest = [&](int arg, const Tensor& p, int bit) -> void* {
      if (!args.need(ctx, arg)) return nullptr;
      if (has_grad_buffer(p, at::kBFloat16, m[2])) {
        acc |= bit;
        return p.grad().data_ptr();
      }
      out[arg] = empty_bf16({r.C}, x);
      return out[arg].data_ptr();
    };
    void *dw = dest(1, w, 1), *db = dest(2, b, 2), *dpc = dest(3, pc, 4), *dpn = nullptr;
    if (args.need(ctx, 4)) {
      out[4] = empty_bf16({r.N, r.C}, x);
      dpn = out[4].data_ptr();
    }
    const float* st = (const float*)stats.data_ptr();
    check(L.eri_gn_bwd(x.data_ptr(), ptr(pc), ptr(pn), dy.data_ptr(), w.data_ptr(), ptr(b), st, st + r.N * G, dx.data_ptr(), dw, db,
                       dpc, dpn, (float*)ws.data_ptr(), r.N, r.HW, r.C, G, (int)m[1], acc, stream()), "gn_bwd");
    out[0] = dx;
    return out;
  }
};

Tensor add_bias_forward(const Tensor& a, const Tensor& b, const Tensor& bias, const Tensor& bias2) {
  const Rows r(a);
  Tensor out = at::empty_like(a);
  check(L.eri_add_bias(a.data_ptr(), b.data_ptr(), ptr(bias), ptr(bias2), out.data_ptr(), (long long)r.N * r.HW, r.C, stream()),
        "add_bias");
  return out;
}
// [N * HW, C] view of a channels-last activation
Tensor as_matrix(const Tensor& x) {
  const Rows r(x);
  return x.dim() == 4 ? x.permute({0, 2, 3, 1}).view({(int64_t)r.N * r.HW, r.C}) : x.view({(int64_t)r.N * r.HW, r.C});
}
struct AddBias : torch::autograd::Function<AddBias> {
  static Tensor forward(AutogradContext* ctx, const OptT& a_o, const OptT& b_o, const OptT& bias_o, const OptT& bias2_o, bool accum) {
    const Tensor a = rows_contig(*a_o), b = rows_contig(*b_o), bias = contig16(opt(bias_o)), bias2 = contig16(opt(bias2_o));
    ctx->saved_data["args"] = Args({&a, &b, &bias, &bias2}).mask;
    ctx->save_for_backward({bias, bias2});
    ctx->saved_data["accum"] = accum;
    return add_bias_forward(a, b, bias, bias2);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto sv = ctx->get_saved_variables();
    const Args args(ctx->saved_data["args"].toInt());
    Tensor d = rows_contig(g[0]);
    variable_list out{d, d, Tensor(), Tensor(), Tensor()};
    for (int i = 0; i < 2; ++i)
      if (args.need(ctx, 2 + i)) out[2 + i] = col_sum(as_matrix(d), sv[i], ctx->saved_data["accum"].toBool());
    return out;
  }
};

struct Upsample2x : torch::autograd::Function<Upsample2x> {
  static Tensor run(const Tensor& x, bool backward) {
    const int64_t N = x.size(0), C = x.size(1), H = backward ? x.size(2) / 2 : x.size(2), W = backward ? x.size(3) / 2 : x.size(3);
    Tensor y = at::empty({N, C, backward ? H : 2 * H, backward ? W : 2 * W}, x.options(), at::MemoryFormat::ChannelsLast);
    check(L.eri_upsample2x(x.data_ptr(), y.data_ptr(), N * H, (int)W, (int)C, backward, stream()), "upsample2x");
    return y;
  }
  static Tensor forward(AutogradContext* ctx, const Tensor& x) { return run(rows_contig(x), false); }
  static variable_list backward(AutogradContext* ctx, variable_list g) { return {run(rows_contig(g[0]), true)}; }
};

}  // namespace

Tensor group_norm_silu(const Tensor& x, const Tensor& w, const OptT& b_, const OptT& pc_, const OptT& pn_, int64_t groups,
                       double eps, bool silu, bool accum) {
  Tensor b = opt(b_), pc = opt(pc_), pn = opt(pn_);
  const Rows r(x);
  check_channels(w, r.C, "group_norm_silu weight");
  check_channels(b, r.C, "group_norm_silu bias");
  check_channels(pc, r.C, "group_norm_silu pre_c");
  if (pn.defined() && pn.dim() == 2 && pn.size(0) == 1 && r.N != 1) pn = pn.expand({r.N, pn.size(1)});   // one embedding for all samples
  check_channels(pn, (int64_t)r.N * r.C, "group_norm_silu pre_nc");
  TORCH_CHECK_VALUE(!pn.defined() || (pn.dim() == 2 && pn.size(0) == r.N), "group_norm_silu pre_nc: ", pn.sizes());
  if (any_grad({&x, &w, &b, &pc, &pn}))
    return GroupNormSilu::apply(wrap(x), wrap(w), wrap(b), wrap(pc), wrap(pn), groups, eps, silu, accum);
  return gn_forward(rows_contig(x), contig16(w), contig16(b), contig16(pc), contig16(pn), groups, eps, silu, Tensor());
}

// a + b + bias + bias2 (per channel): a block's residual sum with the biases of its last convolutions.
Tensor add_bias(const Tensor& a, const Tensor& b, const OptT& bias_, const OptT& bias2_, bool accum) {
  Tensor bias = opt(bias_), bias2 = opt(bias2_);
  const Rows r(a);
  TORCH_CHECK_VALUE(a.sizes() == b.sizes(), "add_bias: ", a.sizes(), " and ", b.sizes());
  check_channels(bias, r.C, "add_bias bias");
  check_channels(bias2, r.C, "add_bias bias2");
  if (any_grad({&a, &b, &bias, &bias2})) return AddBias::apply(wrap(a), wrap(b), wrap(bias), wrap(bias2), accum);
  return add_bias_forward(rows_contig(a), rows_contig(b), contig16(bias), contig16(bias2));
}

// Nearest-neighbour upsampling by two of an [N, C, H, W] activation.
Tensor upsample2x(const Tensor& x) {
  if (any_grad({&x})) return Upsample2x::apply(x);
  return Upsample2x::run(rows_contig(x), false);
}

// Convolution (no bias, one group) with a trained weight in the parameter order [Co, Ci, kh, kw]: the channels-last copy that
// the library reads is made once for both directions, and the weight gradient is added into the parameter's gradient
// in the pass that brings it back into that order.
namespace {
struct TrainedConv : torch::autograd::Function<TrainedConv> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, std::vector<int64_t> strides,
                        std::vector<int64_t> padding, std::vector<int64_t> dilation, bool accum) {
    Tensor rows = at::empty(w.sizes(), w.options(), at::MemoryFormat::ChannelsLast);
    check(L.eri_conv_weight_order(w.data_ptr(), rows.data_ptr(), (int)w.size(0), (int)w.size(1), (int)(w.size(2) * w.size(3)), 0,
                                  stream()), "conv_weight_order");
    ctx->save_for_backward({x, w, rows});
    ctx->saved_data["s"] = strides;
    ctx->saved_data["p"] = padding;
    ctx->saved_data["d"] = dilation;
    ctx->saved_data["accum"] = accum;
    return at::conv2d(x, rows, {}, strides, padding, dilation, 1);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto sv = ctx->get_saved_variables();
    const Tensor &x = sv[0], &w = sv[1], &rows = sv[2];
    const bool nx = ctx->needs_input_grad(0), nw = ctx->needs_input_grad(1);
    auto [dx, dw, db] = at::convolution_backward(g[0], x, rows, std::nullopt, ctx->saved_data["s"].toIntVector(),
                                                 ctx->saved_data["p"].toIntVector(), ctx->saved_data["d"].toIntVector(), false,
                                                 std::vector<int64_t>{0, 0}, 1, {nx, nw, false});
    if (nw && has_grad_buffer(w, at::kBFloat16, ctx->saved_data["accum"].toBool()) && al16(w.grad())) {
      Tensor d = dw.contiguous(at::MemoryFormat::ChannelsLast);
      if (al16(d)) {
        check(L.eri_conv_weight_order(d.data_ptr(), w.grad().data_ptr(), (int)w.size(0), (int)w.size(1),
                                      (int)(w.size(2) * w.size(3)), 1, stream()), "conv_weight_order");
        dw = Tensor();
      }
    }
    return {dx, dw, Tensor(), Tensor(), Tensor(), Tensor()};
  }
};
}  // namespace

Tensor conv2d_trained(const Tensor& x, const Tensor& w, const std::vector<int64_t>& strides, const std::vector<int64_t>& padding,
                      const std::vector<int64_t>& dilation, bool accum) {
  return TrainedConv::apply(x, w, strides, padding, dilation, accum);
}

// ------------------------------------------------------------------------------- FLUX single-stream block
// x + gate * linear2(cat(attn(qkv), gelu(mlp))) where qkv and mlp are column ranges of one projection linear1. The
// column-split epilogue of the GEMM writes both straight to where the next op reads them, and backward produces
// the gradient of the wide projection output in place: the attention columns from the QK-norm / RoPE backward with
// a row stride, the MLP columns from linear2's input-gradient GEMM.
// GELU and its derivative run in an epilogue or as row passes (``flags2`` bits 0 and 1; ops/fused_blocks.py has the
// measurements behind the choice).
namespace {

struct SingleStream : torch::autograd::Function<SingleStream> {
  static Tensor forward(AutogradContext* ctx, const OptT& xm_o, const OptT& x_o, const OptT& gate_o, const OptT& w1_o,
                        const OptT& b1_o, const OptT& w2_o, const OptT& b2_o, const OptT& a1_o, const OptT& bb1_o,
                        const OptT& a2_o, const OptT& bb2_o, const OptT& qs_o, const OptT& ks_o, const OptT& cos_o,
                        const OptT& sin_o, double s1, double s2, int64_t heads, int64_t flags, int64_t flags2, bool keep) {
    const Tensor xm = opt(xm_o), x = opt(x_o), gate = opt(gate_o), w1 = opt(w1_o), b1 = opt(b1_o), w2 = opt(w2_o), b2 = opt(b2_o), a1 = opt(a1_o), bb1 = opt(bb1_o), a2 = opt(a2_o), bb2 = opt(bb2_o), qs = opt(qs_o), ks = opt(ks_o), cos = opt(cos_o), sin = opt(sin_o);
    if (ctx) ctx->saved_data["args"] = Args({&xm, &x, &gate, &w1, &b1, &w2, &b2, &a1, &bb1, &a2, &bb2, &qs, &ks, &cos, &sin}).mask;
    const int64_t B = xm.size(0), Lq = xm.size(1), D = xm.size(2), M = B * Lq, Fm = w1.size(0) - 3 * D, Dh = D / heads;
    Tensor xm2 = contig(xm).view({M, D}), x2 = contig(x).view({M, D}), gate_v = mod_view(gate, D);
    Tensor qkv = empty_bf16({M, 3 * D}, xm), cat = empty_bf16({M, D + Fm}, xm), pre = empty_bf16({M, Fm}, xm);
    Tensor mlp_in = cat.narrow(1, D, Fm), h1, h2;
    const bool pdl = flags & kPdl;
    {
      // each rank-r product is the launch right before the GEMM that consumes it
      if (a1.defined()) h1 = skinny(xm2, a1, (float)s1, (int)flags);
      GemmOpt o;
      o.bias = b1; o.lora_h = h1; o.lora_b = bb1; o.out = qkv; o.n_split = (int)(3 * D); o.pdl = pdl;
      if (flags2 & 1) {
        o.out2 = mlp_in; o.act = 1; o.pre_out = pre;
      } else {
        o.out2 = pre;
      }
      gemm(xm2, w1, o, (int)flags);
      if (!(flags2 & 1))
        check(L.eri_act_fwd_rows(pre.data_ptr(), pre.stride(0), mlp_in.data_ptr(), cat.stride(0), (int)M, (int)Fm, 0, stream()),
              "act_fwd_rows");
    }
    Tensor q = empty_bf16({B, Lq, heads, Dh}, xm), k = at::empty_like(q), v = at::empty_like(q);
    qknorm_fwd(qkv, 3 * D, qs, ks, cos, sin, q, k, v, Lq, 0, 1e-6);
    // the attention writes its output straight into the left column block of the second linear's input
    Tensor o_view = cat.view({B, Lq, D + Fm}).narrow(2, 0, D).unflatten(-1, {heads, Dh});
    Tensor lse = attn_fwd(q, k, v, 1.0 / std::sqrt((double)Dh), o_view, Tensor(), -1).second;
    if (a2.defined()) h2 = skinny(cat, a2, (float)s2, (int)flags);
    GemmOpt o;
    o.bias = b2; o.lora_h = h2; o.lora_b = bb2; o.residual = x2; o.gate = gate_v; o.rows_per_batch = (int)Lq; o.pdl = pdl;
    Tensor y = gemm(cat, w2, o, (int)flags);
    if (keep) {
      ctx->save_for_backward({xm2, qkv, pre, cat, q, k, v, lse, h1, h2, gate_v, w1, w2, a1, bb1, a2, bb2, qs, ks, cos, sin, b1, b2});
      ctx->saved_data["m"] = std::vector<int64_t>{B, Lq, D, Fm, heads, flags, flags2};
      ctx->saved_data["s"] = std::vector<double>{s1, s2};
    }
    return y.view({B, Lq, D});
  }

  static variable_list backward(AutogradContext* ctx, variable_list g_) {
    auto sv = ctx->get_saved_variables();
    const Tensor &xm2 = sv[0], &qkv = sv[1], &pre = sv[2], &cat = sv[3], &q = sv[4], &k = sv[5], &v = sv[6], &lse = sv[7],
                 &h1 = sv[8], &h2 = sv[9], &gate_v = sv[10], &w1 = sv[11], &w2 = sv[12], &a1 = sv[13], &bb1 = sv[14],
                 &a2 = sv[15], &bb2 = sv[16], &qs = sv[17], &ks = sv[18], &cos = sv[19], &sin = sv[20], &b1 = sv[21], &b2 = sv[22];
    const auto m = ctx->saved_data["m"].toIntVector();
    const auto sc = ctx->saved_data["s"].toDoubleVector();
    const int64_t B = m[0], Lq = m[1], D = m[2], Fm = m[3], heads = m[4], Dh = D / heads, M = B * Lq;
    const int flags = (int)m[5];
    const bool pdl = flags & kPdl;
    const Args args(ctx->saved_data["args"].toInt());
    auto need = [&](int i) { return args.need(ctx, i); };
    TORCH_CHECK_NOT_IMPLEMENTED(!need(2), "trainable modulation uses the unfused single-stream path");
    const Tensor& dy = g_[0];
    Tensor o_view = cat.view({B, Lq, D + Fm}).narrow(2, 0, D).unflatten(-1, {heads, Dh});   // the attention's output
    Tensor dy2 = contig(dy).view({M, D});
    Tensor g = gate_rows(Tensor(), dy2, gate_v, Lq);
    Tensor bb2_t, a2_t, bb1_t, a1_t;
    if (a2.defined()) { bb2_t = lora_transposed(bb2); a2_t = lora_transposed(a2); }
    if (a1.defined()) { bb1_t = lora_transposed(bb1); a1_t = lora_transposed(a1); }
    Tensor d_attn = empty_bf16({M, D}, dy), d_h = empty_bf16({M, 3 * D + Fm}, dy), mlp_g = d_h.narrow(1, 3 * D, Fm), ts1, ts2;
    if (a2.defined()) ts2 = skinny(g, bb2_t, (float)sc[1], flags);
    {
      GemmOpt o;
      o.b_mn = true; o.lora_h = ts2; o.lora_b = a2_t; o.out = d_attn; o.n_split = (int)D; o.out2 = mlp_g; o.pdl = pdl;
      if (m[6] & 2) {
        o.act = 3; o.pre_in = pre;
      }
      gemm(g, w2, o, flags);
      if (!(m[6] & 2))
        check(L.eri_act_bwd_rows(mlp_g.data_ptr(), d_h.stride(0), pre.data_ptr(), pre.stride(0), mlp_g.data_ptr(), d_h.stride(0),
                                 (int)M, (int)Fm, 0, stream()), "act_bwd_rows");
    }
    variable_list out(21);
    auto lora = [&](const Tensor& p, const Tensor& at_, const Tensor& bt, bool tr) {
      if (has_grad_buffer(p, at::kBFloat16, flags & kAccumGrad)) return lora_wgrad(at_, bt, p.grad(), tr, true, flags), Tensor();
      return lora_wgrad(at_, bt, Tensor(), tr, false, flags);
    };
    auto dense = [&](const Tensor& p, const Tensor& d, const Tensor& xin) {
      if (has_grad_buffer(p, at::kBFloat16, flags & kAccumGrad)) return wgrad(d, xin, p.grad(), flags), Tensor();
      return wgrad(d, xin, Tensor(), flags);
    };
    if (need(9)) out[9] = lora(a2, cat, ts2, true);
    if (need(10)) out[10] = lora(bb2, g, h2, false);
    auto [dq, dk, dv] = attn_bwd(d_attn.view({B, Lq, heads, Dh}), q, k, v, o_view, lse, 1.0 / std::sqrt((double)Dh), Tensor());
    Tensor dqs = need(11) ? zeros_f32({Dh}, dy) : Tensor();
    Tensor dks = need(12) ? zeros_f32({Dh}, dy) : Tensor();
    check(L.eri_qknorm_rope_bwd(dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), qkv.data_ptr(), ptr(qs), ptr(ks),
                                (const float*)ptr(cos), (const float*)ptr(sin), d_h.data_ptr(), (float*)mptr(dqs),
                                (float*)mptr(dks), (int)B, (int)Lq, (int)heads, (int)Dh, (int)Lq, 0, 1e-6f, (int)(3 * D), (int)D,
                                (int)(3 * D + Fm), stream()), "qknorm_rope_bwd");
    if (a1.defined()) ts1 = skinny(d_h, bb1_t, (float)sc[0], flags);
    if (need(0)) {
      GemmOpt o;
      o.b_mn = true; o.lora_h = ts1; o.lora_b = a1_t; o.pdl = pdl;
      out[0] = gemm(d_h, w1, o, flags).view({B, Lq, D});
    }
    if (need(1)) out[1] = dy;
    if (need(7)) out[7] = lora(a1, xm2, ts1, true);
    if (need(8)) out[8] = lora(bb1, d_h, h1, false);
    if (need(3)) out[3] = dense(w1, d_h, xm2);
    if (need(5)) out[5] = dense(w2, g, cat);
    if (need(4)) out[4] = col_sum(d_h, b1, flags & kAccumGrad);
    if (need(6)) out[6] = col_sum(g, b2, flags & kAccumGrad);
    out[11] = to_bf16(dqs);
    out[12] = to_bf16(dks);
    return out;
  }
};

}  // namespace

Tensor single_stream(const Tensor& xm, const Tensor& x, const Tensor& gate, const Tensor& w1, const OptT& b1,
                     const Tensor& w2, const OptT& b2, const OptT& a1, const OptT& bb1, double s1, const OptT& a2,
                     const OptT& bb2, double s2, const OptT& qs, const OptT& ks, const OptT& cos, const OptT& sin,
                     int64_t heads, int flags, bool act_fwd_epilogue, bool act_bwd_epilogue) {
  const int64_t flags2 = (act_fwd_epilogue ? 1 : 0) | (act_bwd_epilogue ? 2 : 0);
  const Tensor t[] = {opt(b1), opt(b2), opt(a1), opt(bb1), opt(a2), opt(bb2), opt(qs), opt(ks)};
  const Tensor tables[] = {opt(cos), opt(sin)};
  refuse_tangents({&tables[0], &tables[1]});
  const bool keep = any_grad({&xm, &x, &gate, &w1, &w2, &t[0], &t[1], &t[2], &t[3], &t[4], &t[5], &t[6], &t[7]});
  if (!keep)
    return SingleStream::forward(nullptr, xm, x, gate, w1, b1, w2, b2, a1, bb1, a2, bb2, qs, ks, cos, sin,
                                 s1, s2, heads, flags, flags2, false);
  return SingleStream::apply(wrap(xm), wrap(x), wrap(gate), wrap(w1), b1, wrap(w2), b2, a1, bb1, a2, bb2, qs, ks, cos, sin, s1, s2, heads,
                             (int64_t)flags, flags2, true);
}

}  // namespace eri_ops
