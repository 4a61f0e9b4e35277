// Linear layers: act(x W^T + b), LayerNorm(act(x W^T + b)) as one node, LayerNorm.
#include "native.h"

namespace fbn {
namespace {

constexpr int kNone = FB_ACT_NONE;

// The operands of a Linear in the precision of the call: bf16 (cast of x, cached or cast copy of W) or fp32.
struct Operands {
  Tensor x2, w;
  Tensor saved;  // what the backward pass keeps of x: x itself (its version is checked) or the converted copy
};
Operands operands(const Tensor& x, const Tensor& weight, const Tensor& w_low, bool low) {
  TORCH_CHECK_VALUE(weight.is_cuda(), "the weight is not on the input's device");
  Operands o;
  Tensor x2 = as2d(x);
  if (low) {
    o.x2 = is_bf16(x2) ? x2 : cast(x2, at::kBFloat16);
    if (!tma_ok(op2d(o.x2))) o.x2 = contig(o.x2);
    o.w = w_low.defined() ? w_low : cast(weight, at::kBFloat16);
  } else {
    o.x2 = is_f32(x2) ? x2 : cast(x2, at::kFloat);
    o.w = cast(weight, at::kFloat);
  }
  o.saved = o.x2.is_alias_of(x) ? x : o.x2;
  return o;
}

std::vector<int64_t> out_sizes(const Tensor& x, int64_t last) {
  std::vector<int64_t> s(x.sizes().begin(), x.sizes().end());
  s.back() = last;
  return s;
}

// Gradient of a Linear's input, weight and bias from g2 [M, N], in the precision of the forward pass.
void linear_grads(const Tensor& g2, const Tensor& x2, const Tensor& w, bool low, at::ScalarType x_dtype,
                  at::IntArrayRef x_sizes, const std::shared_ptr<Sink>& sink, bool need_x, bool need_w, bool need_b,
                  variable_list& out, const Tensor& sums = Tensor()) {  // sums: the bias' gradient, if known
  const bool tf32 = !low && g_tf32.load(std::memory_order_relaxed);
  const int64_t N = w.size(0), K = w.size(1);
  if (need_x) {  // before the weight gradient: the weight may be overwritten once its bucket is reduced
    Tensor gx = empty(x_sizes, g2, low ? at::kBFloat16 : at::kFloat);
    gemm(op2d(g2), op2d(w).t(), nullptr, kNone, gx.data_ptr(), K, low, false, nullptr, &g2, tf32);
    out[0] = cast(gx, x_dtype);
  }
  if (need_w) {
    if (sink) {
      wgrad_to_sink(*sink, g2, x2);
    } else {
      Tensor gw = empty({N, K}, g2, at::kFloat);
      gemm(op2d(g2).t(), op2d(x2).t(), nullptr, kNone, gw.data_ptr(), K, false, false, nullptr, &g2, tf32, true);
      out[1] = gw;
    }
  }
  if (need_b && sums.defined()) {
    out[2] = sums;
  } else if (need_b) {
    Tensor gb = empty({N}, g2, at::kFloat);
    FB_CALL(fb_colsum, g2.data_ptr(), gb.data_ptr<float>(), g2.size(0), N, dt(g2), 0, cur_stream());
    out[2] = gb;
  }
  if (need_w && sink) sink_ready(*sink);
}

struct LinearNode : Node {
  SavedVariable x_, w_, y_;
  bool low = false, has_bias = false;
  int act = kNone;
  at::ScalarType x_dtype = at::kFloat;
  std::vector<int64_t> x_sizes;
  std::shared_ptr<Sink> sink;
  std::string name() const override { return "FerrumLinearBackward"; }
  void release_variables() override {
    x_.reset_data();
    w_.reset_data();
    y_.reset_data();
  }
  variable_list apply(variable_list&& grads) override {
    variable_list out(3);
    if (!grads[0].defined()) return out;
    Tensor x = x_.unpack(), w = w_.unpack(), y = act != kNone ? y_.unpack(shared_from_this()) : Tensor();
    NoAutograd below;
    Tensor x2 = as2d(x), g2 = contig(as2d(grads[0]));
    g2 = low ? cast(g2, at::kBFloat16) : cast(g2, at::kFloat);
    const bool need_b = has_bias && task_should_compute_output(2);
    Tensor sums;
    if (act != kNone) {  // only activations whose derivative is a function of the output are fused
      y = as2d(y);
      Tensor d = empty(g2.sizes(), g2, g2.scalar_type());
      const uintptr_t at = reinterpret_cast<uintptr_t>(g2.data_ptr()) | reinterpret_cast<uintptr_t>(y.data_ptr()) |
                           reinterpret_cast<uintptr_t>(d.data_ptr());
      // with the bias' gradient, unless its sums want a launch of their own
      if (need_b && g2.numel() > 0 && fb_colsum_clusters(g2.size(0), g2.size(1), dt(g2), 1, at % 16 == 0)) {
        sums = empty({g2.size(1)}, g2, at::kFloat);
        FB_CALL(fb_unary_bwd_colsum, g2.data_ptr(), y.data_ptr(), d.data_ptr(), sums.data_ptr<float>(), g2.size(0), g2.size(1),
                act, dt(g2), cur_stream());
      } else {
        FB_CALL(fb_unary_bwd, g2.data_ptr(), y.data_ptr(), d.data_ptr(), g2.numel(), act, 0.f, 0.f, dt(g2), cur_stream());
      }
      g2 = d;
    }
    linear_grads(g2, x2, w, low, x_dtype, x_sizes, sink, task_should_compute_output(0), task_should_compute_output(1), need_b,
                 out, sums);
    return out;
  }
};

Tensor linear(const Tensor& x, const Tensor& weight, const c10::optional<Tensor>& bias_, int act, bool low, bool tf32,
              const c10::optional<Tensor>& w_low, py::object sink) {
  NoAutograd below;
  const Tensor bias = bias_.value_or(Tensor());
  check_columns(weight, bias, weight.size(0), "the bias");
  Operands o = operands(x, weight, w_low.value_or(Tensor()), low);
  const int64_t N = weight.size(0);
  Tensor y = empty(out_sizes(x, N), o.x2, low ? at::kBFloat16 : at::kFloat);
  Tensor b = bias.defined() ? f32c(bias) : bias;
  const bool grad = wants_grad({&x, &weight, &bias});
  gemm(op2d(o.x2), op2d(o.w), fptr(b), act, y.data_ptr(), N, low, false, nullptr, &o.x2, tf32 && !low);
  if (grad) {
    auto n = make_node<LinearNode>(x, weight, bias);
    n->low = low;
    n->act = act;
    n->has_bias = bias.defined();
    n->x_dtype = x.scalar_type();
    n->x_sizes.assign(x.sizes().begin(), x.sizes().end());
    n->sink = make_sink(sink, py::cast(weight));
    n->x_ = below.keep(o.saved);
    n->w_ = below.keep(o.w);
    torch::autograd::set_history(y, n);
    if (act != kNone) n->y_ = below.keep(y, true);
  }
  return y;
}

// ---------------------------------------------------------------------------------------------- LayerNorm
struct NormStats {
  Tensor mean, rstd;
};
NormStats norm_fwd(const Tensor& x2, const Tensor& gamma, const Tensor& beta, const Tensor& y, float eps, int pre) {
  NormStats s{empty({x2.size(0)}, x2, at::kFloat), empty({x2.size(0)}, x2, at::kFloat)};
  status();  // the wide-row kernels report bounded-wait failures to the status block
  FB_CALL(fb_layernorm_fwd, x2.data_ptr(), fptr(gamma), fptr(beta), y.data_ptr(), s.mean.data_ptr<float>(),
          s.rstd.data_ptr<float>(), x2.size(0), static_cast<int>(x2.size(1)), eps, pre, dt(x2), cur_stream());
  return s;
}
// stats [3, cols]: d_gamma, d_beta, column sum of dx
Tensor norm_bwd(const Tensor& gy2, const Tensor& x2, const Tensor& dact, const Tensor& gamma, const NormStats& s,
                const Tensor& dx, int pre, bool colsum) {
  const int64_t rows = x2.size(0), cols = x2.size(1);
  const int nblk = fb_layernorm_bwd_blocks(rows, static_cast<int>(cols));
  Tensor partial = empty({std::max(nblk, 1), 3, cols}, x2, at::kFloat);
  Tensor stats = empty({3, cols}, x2, at::kFloat);
  FB_CALL(fb_layernorm_bwd, gy2.data_ptr(), x2.data_ptr(), ptr(dact), fptr(gamma), s.mean.data_ptr<float>(),
          s.rstd.data_ptr<float>(), dx.data_ptr(), partial.data_ptr<float>(), stats.data_ptr<float>(), rows,
          static_cast<int>(cols), pre, dt(x2), nblk, colsum ? 3 : 2, cur_stream());
  return stats;
}

struct LayerNormNode : Node {
  SavedVariable x_, g_, mean_, rstd_;
  int pre = kNone;
  bool has_gamma = false, has_beta = false;
  std::string name() const override { return "FerrumLayerNormBackward"; }
  void release_variables() override {
    x_.reset_data();
    g_.reset_data();
    mean_.reset_data();
    rstd_.reset_data();
  }
  variable_list apply(variable_list&& grads) override {
    variable_list out(3);
    if (!grads[0].defined()) return out;
    Tensor x = x_.unpack(), g = g_.unpack();
    const NormStats st{mean_.unpack(), rstd_.unpack()};
    NoAutograd below;
    x = contig(x);
    Tensor x2 = as2d(x), gy = contig(cast(grads[0], x.scalar_type()));
    Tensor dx = empty(x.sizes(), x, x.scalar_type());
    Tensor stats = norm_bwd(as2d(gy), x2, Tensor(), g, st, dx, pre, false);
    out[0] = dx;
    if (has_gamma) out[1] = stats[0];
    if (has_beta) out[2] = stats[1];
    return out;
  }
};

// The normalisation kernels evaluate a GELU in front of the statistics; any other activation is an op of its own.
bool norm_evaluates(int act) { return act == kNone || act == FB_ACT_GELU; }

Tensor layer_norm(const Tensor& x, const c10::optional<Tensor>& gamma_, const c10::optional<Tensor>& beta_, double eps,
                  int pre) {
  if (!norm_evaluates(pre)) return layer_norm(unary(x, pre, 0., 0.), gamma_, beta_, eps, kNone);
  NoAutograd below;
  const Tensor gamma = gamma_.value_or(Tensor()), beta = beta_.value_or(Tensor());
  check_columns(x, gamma, x.size(-1), "the scale");
  check_columns(x, beta, x.size(-1), "the shift");
  Tensor xc = contig(x);
  Tensor g = gamma.defined() ? contig(gamma) : gamma, b = beta.defined() ? contig(beta) : beta;
  Tensor y = empty(xc.sizes(), xc, xc.scalar_type());
  NormStats st = norm_fwd(as2d(xc), g, b, as2d(y), static_cast<float>(eps), pre);
  if (wants_grad({&x, &gamma, &beta})) {
    auto n = make_node<LayerNormNode>(x, gamma, beta);
    n->mean_ = below.keep(st.mean);
    n->rstd_ = below.keep(st.rstd);
    n->pre = pre;
    n->has_gamma = gamma.defined();
    n->has_beta = beta.defined();
    n->x_ = below.keep(xc.is_alias_of(x) ? x : xc);
    n->g_ = below.keep(g);
    torch::autograd::set_history(y, n);
  }
  return y;
}

// ---------------------------------------------------------------- LayerNorm(x + r) as one node
// The residual connection of fp32 activations: the addition goes along with the normalisation, and the backward kernel
// writes the gradient of a bf16 branch beside the fp32 one.
struct AddNormNode : Node {
  SavedVariable sum_, g_, mean_, rstd_;
  bool has_beta = false, has_gamma = false;
  at::ScalarType r_dtype = at::kFloat;
  std::string name() const override { return "FerrumAddLayerNormBackward"; }
  void release_variables() override {
    for (SavedVariable* s : {&sum_, &g_, &mean_, &rstd_}) s->reset_data();
  }
  variable_list apply(variable_list&& grads) override {
    variable_list out(4);  // x, r, gamma, beta
    if (!grads[0].defined()) return out;
    Tensor sum = sum_.unpack(), g = g_.unpack(), mean = mean_.unpack(), rstd = rstd_.unpack();
    NoAutograd below;
    sum = contig(sum);
    Tensor s2 = as2d(sum), gy = f32c(grads[0]), dx = empty(sum.sizes(), sum, at::kFloat), low;
    if (r_dtype == at::kBFloat16 && task_should_compute_output(1)) low = empty(sum.sizes(), sum, at::kBFloat16);
    const int64_t rows = s2.size(0), cols = s2.size(1);
    Tensor stats;
    if (low.defined() && reinterpret_cast<uintptr_t>(gy.data_ptr()) % 16 == 0 &&
        reinterpret_cast<uintptr_t>(sum.data_ptr()) % 16 == 0 && (!g.defined() || reinterpret_cast<uintptr_t>(g.data_ptr()) % 16 == 0)) {
      const int nblk = fb_layernorm_bwd_blocks(rows, static_cast<int>(cols));
      Tensor partial = empty({std::max(nblk, 1), 3, cols}, sum, at::kFloat);
      stats = empty({3, cols}, sum, at::kFloat);
      FB_CALL(fb_add_layernorm_bwd, gy.data_ptr<float>(), sum.data_ptr<float>(), fptr(g), mean.data_ptr<float>(),
              rstd.data_ptr<float>(), dx.data_ptr<float>(), low.data_ptr(), partial.data_ptr<float>(),
              stats.data_ptr<float>(), rows, static_cast<int>(cols), nblk, cur_stream());
      out[1] = low;
    } else {
      stats = norm_bwd(as2d(gy), s2, Tensor(), g, NormStats{mean, rstd}, dx, kNone, false);
      if (task_should_compute_output(1)) out[1] = cast(dx, r_dtype);
    }
    out[0] = dx;
    if (has_gamma) out[2] = stats[0];
    if (has_beta) out[3] = stats[1];
    return out;
  }
};

Tensor add_layer_norm(const Tensor& x, const Tensor& r, const c10::optional<Tensor>& gamma_,
                      const c10::optional<Tensor>& beta_, double eps) {
  const Tensor gamma = gamma_.value_or(Tensor()), beta = beta_.value_or(Tensor());
  const int64_t cols = x.dim() > 0 ? x.size(-1) : 0;
  const auto f32 = [&](const Tensor& t) { return !t.defined() || (t.scalar_type() == at::kFloat && t.is_cuda() && t.numel() == cols); };
  const bool whole = x.scalar_type() == at::kFloat && (r.scalar_type() == at::kFloat || is_bf16(r)) &&
                     x.sizes() == r.sizes() && x.device() == r.device() && x.numel() > 0 && cols % 8 == 0 && cols <= 8192 &&
                     f32(gamma) && f32(beta);
  Tensor y;
  if (whole) {
    NoAutograd below;
    Tensor xc = contig(x), rc = contig(r), g = gamma.defined() ? contig(gamma) : gamma, b = beta.defined() ? contig(beta) : beta;
    uintptr_t at = reinterpret_cast<uintptr_t>(xc.data_ptr()) | reinterpret_cast<uintptr_t>(rc.data_ptr());
    for (const Tensor& t : {g, b})
      if (t.defined()) at |= reinterpret_cast<uintptr_t>(t.data_ptr());
    if (at % 16 == 0) {
      const bool grad = wants_grad({&x, &r, &gamma, &beta});
      const int64_t rows = xc.numel() / cols;
      Tensor sum = grad ? empty(xc.sizes(), xc, at::kFloat) : Tensor();
      NormStats st{empty({rows}, xc, at::kFloat), empty({rows}, xc, at::kFloat)};
      y = empty(xc.sizes(), xc, at::kFloat);
      FB_CALL(fb_add_layernorm_fwd, xc.data_ptr<float>(), rc.data_ptr(), fptr(g), fptr(b), static_cast<float*>(ptr(sum)), y.data_ptr<float>(),
              st.mean.data_ptr<float>(), st.rstd.data_ptr<float>(), rows, static_cast<int>(cols), static_cast<float>(eps),
              dt(rc), cur_stream());
      if (grad) {
        auto n = make_node<AddNormNode>(x, r, gamma, beta);
        n->has_gamma = gamma.defined();
        n->has_beta = beta.defined();
        n->r_dtype = r.scalar_type();
        n->sum_ = below.keep(sum);
        n->g_ = below.keep(g);
        n->mean_ = below.keep(st.mean);
        n->rstd_ = below.keep(st.rstd);
        torch::autograd::set_history(y, n);
      }
      return y;
    }
  }
  return layer_norm(fbn::add(x, r), gamma_, beta_, eps, kNone);
}

// ---------------------------------------------------------------- LayerNorm(act(x W^T + b)) as one node
// Tensor-core path: the GEMM epilogue writes act(z) and, where a backward pass follows, act'(z); the normalisation
// reads act(z).  Backward: one streaming kernel turns dy into dz and yields d_gamma, d_beta and the bias gradient,
// then the two products run on dz.  fp32 path: z is stored, the activation is evaluated inside the normalisation.
struct LinearActNormNode : Node {
  SavedVariable x_, w_, g_, z_, dact_, mean_, rstd_;
  bool low = false, has_bias = false;
  int pre = kNone;
  at::ScalarType x_dtype = at::kFloat;
  std::vector<int64_t> x_sizes;
  std::shared_ptr<Sink> sink;
  std::string name() const override { return "FerrumLinearActNormBackward"; }
  void release_variables() override {
    for (SavedVariable* s : {&x_, &w_, &g_, &z_, &dact_, &mean_, &rstd_}) s->reset_data();
  }
  variable_list apply(variable_list&& grads) override {
    variable_list out(5);
    if (!grads[0].defined()) return out;
    Tensor x = x_.unpack(), w = w_.unpack(), g = g_.unpack(), z = z_.unpack(), dact = dact_.unpack();
    const NormStats st{mean_.unpack(), rstd_.unpack()};
    NoAutograd below;
    Tensor x2 = as2d(x);
    Tensor gy2 = contig(as2d(cast(grads[0], z.scalar_type())));
    Tensor dz = empty(z.sizes(), z, z.scalar_type());
    Tensor stats = norm_bwd(gy2, z, dact, g, st, dz, pre, true);
    linear_grads(dz, x2, w, low, x_dtype, x_sizes, sink, task_should_compute_output(0), task_should_compute_output(1),
                 false, out);
    if (has_bias) out[2] = stats[2];
    out[3] = stats[0];
    out[4] = stats[1];
    return out;
  }
};

Tensor linear_act_norm(const Tensor& x, const Tensor& weight, const c10::optional<Tensor>& bias_, const Tensor& gamma,
                       const Tensor& beta, double eps, int act, bool low, bool tf32,
                       const c10::optional<Tensor>& w_low, py::object sink) {
  if (!low && !norm_evaluates(act))
    return layer_norm(linear(x, weight, bias_, kNone, low, tf32, w_low, sink), gamma, beta, eps, act);
  const Tensor bias = bias_.value_or(Tensor());
  check_columns(weight, bias, weight.size(0), "the bias");
  check_columns(weight, gamma, weight.size(0), "the scale");
  check_columns(weight, beta, weight.size(0), "the shift");
  Operands o;
  {
    NoAutograd below;
    o = operands(x, weight, w_low.value_or(Tensor()), low);
  }
  const bool fused = low && act != kNone && tma_ok(op2d(o.x2)) && tma_ok(op2d(o.w));
  if (fused && act > FB_ACT_SIGMOID) throw py::key_error("linear_act_layernorm: an activation that no epilogue evaluates");
  if (!fused && !norm_evaluates(act))
    return layer_norm(linear(x, weight, bias_, kNone, low, tf32, w_low, sink), gamma, beta, eps, act);
  NoAutograd below;
  const int64_t N = weight.size(0), M = o.x2.size(0);
  const bool grad = wants_grad({&x, &weight, &bias, &gamma, &beta});
  Tensor b = bias.defined() ? f32c(bias) : bias;
  Tensor g = contig(gamma), be = contig(beta);
  Tensor z = empty({M, N}, o.x2, low ? at::kBFloat16 : at::kFloat), dact;
  if (fused && grad) dact = empty({M, N}, o.x2, at::kBFloat16);
  gemm(op2d(o.x2), op2d(o.w), fptr(b), fused ? act : kNone, z.data_ptr(), N, low, false, ptr(dact), &o.x2,
       tf32 && !low);
  const int pre = fused ? kNone : act;
  Tensor y = empty(out_sizes(x, N), o.x2, z.scalar_type());
  NormStats st = norm_fwd(z, g, be, y, static_cast<float>(eps), pre);
  if (grad) {
    auto n = make_node<LinearActNormNode>(x, weight, bias, gamma, beta);
    n->low = low;
    n->pre = pre;
    n->has_bias = bias.defined();
    n->x_dtype = x.scalar_type();
    n->x_sizes.assign(x.sizes().begin(), x.sizes().end());
    n->sink = make_sink(sink, py::cast(weight));
    n->x_ = below.keep(o.saved);
    n->w_ = below.keep(o.w);
    n->g_ = below.keep(g);
    n->z_ = below.keep(z);
    n->dact_ = below.keep(dact);
    n->mean_ = below.keep(st.mean);
    n->rstd_ = below.keep(st.rstd);
    torch::autograd::set_history(y, n);
  }
  return y;
}

// ------------------------------------------------------------------------------------- batched products
// alpha * a b for [Bo, Bi, M, K] x [Bo, Bi, K, N] views (heads interleaved in the feature dimension, transposes):
// fp32 operands on the fp32 tensor-core kernel with any strides, bf16 ones through 4-D TMA maps.
bool batched_tma_ok(const Tensor& t) {
  if (reinterpret_cast<uintptr_t>(t.data_ptr()) % 16) return false;
  const ll s0 = t.stride(2), s1 = t.stride(3);
  ll ld;
  if (s1 == 1) ld = s0 >= t.size(3) ? s0 : 1;
  else if (s0 == 1) ld = s1 >= t.size(2) ? s1 : 1;
  else return false;
  if (ld % 8) return false;
  for (int d = 0; d < 2; ++d)
    if (t.size(d) != 1 && (t.stride(d) <= 0 || t.stride(d) % 8)) return false;
  return true;
}
Tensor batched_operand(const Tensor& t, bool low) {
  if (!low) return cast(t, at::kFloat);
  Tensor b = cast(t, at::kBFloat16);
  return batched_tma_ok(b) ? b : b.contiguous();
}
// out = alpha * a b^T with a [.., M, K], b [.., N, K]
void batched_nt(const Tensor& a, const Tensor& b, const Tensor& out, float alpha) {
  const int M = static_cast<int>(a.size(2)), N = static_cast<int>(b.size(2)), K = static_cast<int>(a.size(3));
  const int Bo = static_cast<int>(a.size(0)), Bi = static_cast<int>(a.size(1));
  if (is_f32(a)) {
    FB_CALL(fb_gemm_f32_tensor, a.data_ptr<float>(), b.data_ptr<float>(), out.data_ptr<float>(), nullptr, M, N, K,
            a.stride(2), a.stride(3), b.stride(2), b.stride(3), out.stride(2), 0, 0, alpha, Bo, Bi, a.stride(0),
            a.stride(1), b.stride(0), b.stride(1), out.stride(0), out.stride(1), status(), cur_stream());
    return;
  }
  const int a_mn = a.stride(3) == 1 ? 0 : 1, b_mn = b.stride(3) == 1 ? 0 : 1;
  FB_CALL(fb_gemm_bf16_batched, a.data_ptr(), b.data_ptr(), out.data_ptr(), M, N, K, a_mn ? a.stride(3) : a.stride(2),
          b_mn ? b.stride(3) : b.stride(2), out.stride(2), Bo, Bi, a.stride(0), a.stride(1), b.stride(0), b.stride(1),
          out.stride(0), out.stride(1), a_mn, b_mn, 1, 0, alpha, status(), cur_stream());
}
Tensor batched_usable(const Tensor& t) { return is_f32(t) || batched_tma_ok(t) ? t : t.contiguous(); }

struct BmmNode : Node {
  SavedVariable a_, b_;
  float alpha = 1.f;
  at::ScalarType da = at::kFloat, db = at::kFloat;
  std::string name() const override { return "FerrumBmmBackward"; }
  void release_variables() override {
    a_.reset_data();
    b_.reset_data();
  }
  variable_list apply(variable_list&& grads) override {
    variable_list out(2);
    if (!grads[0].defined()) return out;
    Tensor a = a_.unpack(), b = b_.unpack();
    NoAutograd below;
    Tensor g = batched_operand(grads[0], is_bf16(a));
    if (task_should_compute_output(0)) {
      Tensor ga = empty(a.sizes(), a, a.scalar_type());
      batched_nt(g, b, ga, alpha);
      out[0] = cast(ga, da);
    }
    if (task_should_compute_output(1)) {
      Tensor gb = empty(b.sizes(), b, b.scalar_type());
      batched_nt(a.transpose(-1, -2), g.transpose(-1, -2), gb, alpha);
      out[1] = cast(gb, db);
    }
    return out;
  }
};

Tensor bmm(const Tensor& a, const Tensor& b, double alpha, bool heads_inner, bool low) {
  NoAutograd below;
  TORCH_CHECK_VALUE(a.dim() == 4 && b.dim() == 4 && a.size(0) == b.size(0) && a.size(1) == b.size(1) &&
                        a.size(3) == b.size(2),
                    "bmm: [Bo, Bi, M, K] x [Bo, Bi, K, N] expected, got ", a.sizes(), " x ", b.sizes());
  Tensor ac = batched_operand(a, low), bc = batched_operand(b, low);
  const auto st = low ? at::kBFloat16 : at::kFloat;
  const int64_t Bo = a.size(0), Bi = a.size(1), M = a.size(2), N = b.size(3);
  // heads_inner: stored [Bo, M, Bi, N], so that merging the heads afterwards is a view
  Tensor y = heads_inner ? empty({Bo, M, Bi, N}, ac, st).permute({0, 2, 1, 3}) : empty({Bo, Bi, M, N}, ac, st);
  if (y.numel() > 0) batched_nt(ac, batched_usable(bc.transpose(-1, -2)), y, static_cast<float>(alpha));
  if (wants_grad({&a, &b})) {
    auto n = make_node<BmmNode>(a, b);
    n->alpha = static_cast<float>(alpha);
    n->da = a.scalar_type();
    n->db = b.scalar_type();
    n->a_ = below.keep(ac);
    n->b_ = below.keep(bc);
    torch::autograd::set_history(y, n);
  }
  return y;
}

}  // namespace

void bind_linear(py::module_& m) {
  m.def("linear", &linear);
  m.def("layer_norm", &layer_norm);
  m.def("add_layer_norm", &add_layer_norm);
  m.def("linear_act_norm", &linear_act_norm);
  m.def("bmm", &bmm);
  m.def("low_copy", [](const Tensor& x) {  // bf16 copy, without a graph, for several products; a dual tensor is refused
    refuse_tangents({&x});
    NoAutograd below;
    return cast(x, at::kBFloat16);
  });
  m.def("gemm_nt",  // out = act(a b^T + bias) without a graph; see ops/functional.py
        [](const Tensor& a, const Tensor& b, const c10::optional<Tensor>& bias, int act, const Tensor& out,
           bool accumulate, bool tf32) {
          Tensor bb = bias.has_value() ? *bias : Tensor();
          gemm(op2d(a), op2d(b), fptr(bb), act, out.data_ptr(), out.stride(0), is_bf16(out), accumulate, nullptr, &out,
               tf32);
        });
}

}  // namespace fbn
