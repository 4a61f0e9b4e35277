// Unary and binary ops, softmax, losses.
#include "native.h"

namespace fbn {
namespace {

bool saves_output(int op) { return op == FB_ACT_TANH || op == FB_ACT_SIGMOID || op == FB_UNARY_EXP || op == FB_UNARY_SQRT; }
bool saves_nothing(int op) {
  return op == FB_ACT_NONE || op == FB_UNARY_NEG || op == FB_UNARY_ADD_SCALAR || op == FB_UNARY_MUL_SCALAR ||
         op == FB_UNARY_RSUB_SCALAR || op == FB_UNARY_AFFINE;
}

struct UnaryNode : Node {
  SavedVariable s_;
  int op = 0;
  float alpha = 0.f, beta = 0.f;
  std::string name() const override { return "FerrumUnaryBackward"; }
  void release_variables() override { s_.reset_data(); }
  variable_list apply(variable_list&& grads) override {
    variable_list out(1);
    if (!grads[0].defined()) return out;
    Tensor s;
    if (!saves_nothing(op)) s = s_.unpack(saves_output(op) ? shared_from_this() : nullptr);
    NoAutograd below;
    Tensor g = contig(grads[0]);
    if (s.defined()) s = cast(contig(s), g.scalar_type());
    Tensor dx = empty(g.sizes(), g, g.scalar_type());
    FB_CALL(fb_unary_bwd, g.data_ptr(), ptr(s), dx.data_ptr(), g.numel(), op, alpha, beta, dt(g), cur_stream());
    out[0] = dx;
    return out;
  }
};

}  // namespace

Tensor unary(const Tensor& x, int op, double alpha, double beta) {
  NoAutograd below;
  Tensor xc = contig(x), y = empty(x.sizes(), x, x.scalar_type());
  FB_CALL(fb_unary_fwd, xc.data_ptr(), y.data_ptr(), xc.numel(), op, static_cast<float>(alpha),
          static_cast<float>(beta), dt(xc), cur_stream());
  if (wants_grad({&x})) {
    auto n = make_node<UnaryNode>(x);
    n->op = op;
    n->alpha = static_cast<float>(alpha);
    n->beta = static_cast<float>(beta);
    torch::autograd::set_history(y, n);
    if (saves_output(op)) n->s_ = below.keep(y, true);
    else if (!saves_nothing(op)) n->s_ = below.keep(x);
  }
  return y;
}

namespace {

// Same-shape add, the residual connection: fp32 result of any mix of fp32 and bf16 operands (bf16 of two bf16 ones).
struct AddNode : Node {
  at::ScalarType da = at::kFloat, db = at::kFloat;
  std::string name() const override { return "FerrumAddBackward"; }
  variable_list apply(variable_list&& grads) override {
    NoAutograd below;
    variable_list out(2);
    if (!grads[0].defined()) return out;
    if (task_should_compute_output(0)) out[0] = cast(grads[0], da);
    if (task_should_compute_output(1)) out[1] = da == db && out[0].defined() ? out[0] : cast(grads[0], db);
    return out;
  }
};

}  // namespace
Tensor add(const Tensor& a, const Tensor& b) {
  NoAutograd below;
  Tensor ac = f32c(a), bc = f32c(b), y = empty(a.sizes(), a, at::kFloat);
  const ll n = y.numel(), one = 1;
  FB_CALL(fb_binary_fwd, ac.data_ptr<float>(), bc.data_ptr<float>(), y.data_ptr<float>(), FB_BIN_ADD, 1, &n, &one, &one,
          cur_stream());
  if (is_bf16(a) && is_bf16(b)) y = cast(y, at::kBFloat16);
  if (wants_grad({&a, &b})) {
    auto nd = make_node<AddNode>(a, b);
    nd->da = a.scalar_type();
    nd->db = b.scalar_type();
    torch::autograd::set_history(y, nd);
  }
  return y;
}
namespace {

// ------------------------------------------------------------------------------------------------- softmax
struct SoftmaxNode : Node {
  SavedVariable y_;
  int log_mode = 0;
  std::string name() const override { return "FerrumSoftmaxBackward"; }
  void release_variables() override { y_.reset_data(); }
  variable_list apply(variable_list&& grads) override {
    variable_list out(1);
    if (!grads[0].defined()) return out;
    Tensor y = y_.unpack(shared_from_this());
    NoAutograd below;
    Tensor g = contig(cast(grads[0], y.scalar_type())), dx = empty(y.sizes(), y, y.scalar_type());
    FB_CALL(fb_softmax_bwd, g.data_ptr(), y.data_ptr(), dx.data_ptr(), rows_of(y), static_cast<int>(y.size(-1)),
            log_mode, dt(y), cur_stream());
    out[0] = dx;
    return out;
  }
};

Tensor softmax(const Tensor& x, bool log_mode) {
  NoAutograd below;
  Tensor xc = contig(x), y = empty(x.sizes(), x, x.scalar_type());
  FB_CALL(fb_softmax_fwd, xc.data_ptr(), y.data_ptr(), rows_of(xc), static_cast<int>(xc.size(-1)), log_mode, dt(xc),
          cur_stream());
  if (wants_grad({&x})) {
    auto n = make_node<SoftmaxNode>(x);
    n->log_mode = log_mode;
    torch::autograd::set_history(y, n);
    n->y_ = below.keep(y, true);
  }
  return y;
}

// -------------------------------------------------------------------------------------------------- losses
// Mean cross-entropy of logits and integer labels.  The forward pass writes the logit gradient of a unit loss, the
// backward pass multiplies it by the incoming gradient (read on the device).
struct CrossEntropyNode : Node {
  SavedVariable dx_, labels_;  // labels: saved, so that labels changed before the backward pass are noticed
  std::string name() const override { return "FerrumCrossEntropyBackward"; }
  void release_variables() override {
    dx_.reset_data();
    labels_.reset_data();
  }
  variable_list apply(variable_list&& grads) override {
    variable_list out(1);
    if (!grads[0].defined()) return out;
    labels_.unpack();
    Tensor dx = dx_.unpack();
    NoAutograd below;
    Tensor g = f32c(grads[0]), y = empty(dx.sizes(), dx, dx.scalar_type());
    FB_CALL(fb_scale_by_device_scalar, dx.data_ptr(), g.data_ptr<float>(), y.data_ptr(), dx.numel(), dt(dx), cur_stream());
    out[0] = y;
    return out;
  }
};

Tensor cross_entropy(const Tensor& logits, const Tensor& labels) {
  NoAutograd below;
  TORCH_CHECK_VALUE(logits.dim() == 2 && labels.numel() == logits.size(0),
                    "cross_entropy: one label per row expected, got ", labels.sizes(), " for ", logits.sizes());
  TORCH_CHECK_VALUE(logits.numel() > 0, "cross_entropy: no mean over an empty batch, got ", logits.sizes());
  check_on(logits, labels, "the label tensor");
  Tensor x = contig(logits), lab = contig(labels);
  const int64_t rows = x.size(0);
  const bool grad = wants_grad({&logits});
  Tensor loss = empty({}, x, at::kFloat), dx = grad ? empty(x.sizes(), x, x.scalar_type()) : Tensor();
  Tensor ws = empty({fb_mean_loss_workspace(rows)}, x, at::kFloat);
  FB_CALL(fb_ce_fwd, x.data_ptr(), reinterpret_cast<const ll*>(lab.data_ptr<int64_t>()), ptr(dx), loss.data_ptr<float>(),
          ws.data_ptr<float>(), rows, static_cast<int>(x.size(1)), 1.f / static_cast<float>(rows), dt(x), cur_stream());
  if (grad) {
    auto n = make_node<CrossEntropyNode>(logits);
    n->dx_ = below.keep(dx);
    n->labels_ = below.keep(lab);
    torch::autograd::set_history(loss, n);
  }
  return loss;
}

// Mean of -log_probs[i, target_i].
struct NllNode : Node {
  SavedVariable target_;
  int64_t rows = 0, cols = 0;
  at::ScalarType st = at::kFloat;
  std::vector<int64_t> sizes;
  std::string name() const override { return "FerrumNllBackward"; }
  void release_variables() override { target_.reset_data(); }
  variable_list apply(variable_list&& grads) override {
    variable_list out(1);
    if (!grads[0].defined()) return out;
    Tensor target = target_.unpack();
    NoAutograd below;
    Tensor g = f32c(grads[0]), dx = empty(sizes, g, st);
    FB_CALL(fb_nll_bwd, reinterpret_cast<const ll*>(target.data_ptr<int64_t>()), g.data_ptr<float>(), dx.data_ptr(),
            rows, static_cast<int>(cols), -1.f / static_cast<float>(rows), dt(dx), cur_stream());
    out[0] = dx;
    return out;
  }
};

// Whether the op takes these arguments: one target per row, on the device of the log-probabilities.
bool nll_takes(const Tensor& log_probs, const Tensor& target) {
  return log_probs.is_cuda() && (is_f32(log_probs) || is_bf16(log_probs)) && log_probs.numel() > 0 &&
         target.numel() == rows_of(log_probs) && target.device() == log_probs.device();
}
Tensor nll(const Tensor& log_probs, const Tensor& target) {
  NoAutograd below;
  const int64_t cols = log_probs.size(-1), rows = rows_of(log_probs);
  TORCH_CHECK_VALUE(rows > 0 && target.numel() == rows, "nll: one target per row expected, got ", target.sizes(), " for ",
                    log_probs.sizes());
  check_on(log_probs, target, "the target");
  Tensor x = contig(log_probs), t = contig(target.scalar_type() == at::kLong ? target : target.to(at::kLong));
  Tensor loss = empty({}, x, at::kFloat), ws = empty({fb_mean_loss_workspace(rows)}, x, at::kFloat);
  FB_CALL(fb_nll_fwd, x.data_ptr(), reinterpret_cast<const ll*>(t.data_ptr<int64_t>()), loss.data_ptr<float>(),
          ws.data_ptr<float>(), rows, static_cast<int>(cols), -1.f / static_cast<float>(rows), dt(x), status(), cur_stream());
  if (!is_f32(x)) loss = cast(loss, x.scalar_type());
  if (wants_grad({&log_probs})) {
    auto n = make_node<NllNode>(log_probs);
    n->target_ = below.keep(t);
    n->rows = rows;
    n->cols = cols;
    n->st = x.scalar_type();
    n->sizes.assign(x.sizes().begin(), x.sizes().end());
    torch::autograd::set_history(loss, n);
  }
  return loss;
}

// mse / bce / l1 / smooth_l1, mean over all elements; predictions fp32 or bf16, targets likewise.
struct ElemLossNode : Node {
  SavedVariable p_, t_;  // as the kernels read them: the arguments themselves only where they were not converted
  int kind = 0;
  at::ScalarType st = at::kFloat;
  std::string name() const override { return "FerrumElementwiseLossBackward"; }
  void release_variables() override {
    p_.reset_data();
    t_.reset_data();
  }
  variable_list apply(variable_list&& grads) override {
    variable_list out(1);
    if (!grads[0].defined()) return out;
    Tensor p = p_.unpack(), t = t_.unpack();
    NoAutograd below;
    Tensor g = f32c(grads[0]), dp = empty(p.sizes(), p, at::kFloat);
    FB_CALL(fb_loss_bwd, p.data_ptr<float>(), t.data_ptr<float>(), g.data_ptr<float>(), dp.data_ptr<float>(), p.numel(),
            kind, 1.f / static_cast<float>(p.numel()), cur_stream());
    out[0] = cast(dp, st);
    return out;
  }
};

Tensor elementwise_loss(const Tensor& pred, const Tensor& target, int kind) {
  NoAutograd below;
  TORCH_CHECK_VALUE(pred.sizes() == target.sizes(), "loss: predictions ", pred.sizes(), " and targets ", target.sizes());
  check_on(pred, target, "the target");
  refuse_tangents({&target});
  Tensor p = f32c(pred), t = f32c(target);
  const int64_t n = p.numel();
  Tensor loss = empty({}, p, at::kFloat), ws = empty({fb_mean_loss_workspace(n)}, p, at::kFloat);
  FB_CALL(fb_loss_mean_fwd, p.data_ptr<float>(), t.data_ptr<float>(), loss.data_ptr<float>(), ws.data_ptr<float>(), n,
          kind, 1.f / static_cast<float>(n), cur_stream());
  if (wants_grad({&pred})) {
    auto nd = make_node<ElemLossNode>(pred);
    nd->p_ = below.keep(p);
    nd->t_ = below.keep(t);
    nd->kind = kind;
    nd->st = pred.scalar_type();
    torch::autograd::set_history(loss, nd);
  }
  return loss;
}

}  // namespace

void bind_elementwise(py::module_& m) {
  m.def("unary", &unary);
  m.def("add", &add);
  m.def("softmax", &softmax);
  m.def("cross_entropy", &cross_entropy);
  m.def("nll", &nll);
  m.def("nll_takes", &nll_takes);
  m.def("elementwise_loss", &elementwise_loss);
}

}  // namespace fbn
