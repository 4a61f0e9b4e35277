// Ungrouped 2-D convolutions under bf16 autocast as implicit GEMMs (gemm/tcgen05_gemm.cu, conv forms): act(conv(x, w, b))
// or conv(x, w, b) + add as one node.  NCHW fp32 in and out; between the layout kernels of kernels/conv_layout.cu
// everything is NHWC, bf16 where it is an operand.
#include "native.h"

namespace fbn {
namespace {

// The convolution as the implicit GEMM sees it: stride 1 over z (see kernels/conv_layout.cu).
struct Shape {
  int B, C, H, W, O, kh, kw, sh, sw, ph, pw, dh, dw;
  int Ho, Wo;
  bool strided;
  int eh, ew, k2h, k2w, Hz, Wz, Cz, Op;
  int lph, lpw;  // padding written into z
  int gph, gpw;  // padding left to the GEMM's zero fill
};
int pad8(int n) { return (n + 7) / 8 * 8; }
Shape shape_of(at::IntArrayRef x, at::IntArrayRef w, at::IntArrayRef stride, at::IntArrayRef padding, at::IntArrayRef dilation) {
  Shape s;
  s.B = static_cast<int>(x[0]); s.C = static_cast<int>(x[1]); s.H = static_cast<int>(x[2]); s.W = static_cast<int>(x[3]);
  s.O = static_cast<int>(w[0]); s.kh = static_cast<int>(w[2]); s.kw = static_cast<int>(w[3]);
  s.sh = static_cast<int>(stride[0]); s.sw = static_cast<int>(stride[1]);
  s.ph = static_cast<int>(padding[0]); s.pw = static_cast<int>(padding[1]);
  s.dh = static_cast<int>(dilation[0]); s.dw = static_cast<int>(dilation[1]);
  s.Ho = (s.H + 2 * s.ph - s.dh * (s.kh - 1) - 1) / s.sh + 1;
  s.Wo = (s.W + 2 * s.pw - s.dw * (s.kw - 1) - 1) / s.sw + 1;
  s.strided = s.sh != 1 || s.sw != 1;
  s.eh = std::min(s.sh, s.kh);
  s.ew = std::min(s.sw, s.kw);
  s.k2h = (s.kh + s.sh - 1) / s.sh;
  s.k2w = (s.kw + s.sw - 1) / s.sw;
  s.Hz = s.strided ? s.Ho + s.k2h - 1 : s.H;
  s.Wz = s.strided ? s.Wo + s.k2w - 1 : s.W;
  s.Cz = pad8(s.eh * s.ew * s.C);
  s.Op = pad8(s.O);
  s.lph = s.strided ? s.ph : 0;
  s.lpw = s.strided ? s.pw : 0;
  s.gph = s.strided ? 0 : s.ph;
  s.gpw = s.strided ? 0 : s.pw;
  return s;
}

Tensor packed_filters(const Tensor& w, const Shape& s, bool dgrad) {
  const int rows = dgrad ? s.eh * s.ew * s.C : s.O, pitch = dgrad ? s.Op : s.Cz;
  Tensor out = empty({rows, s.k2h * s.k2w, pitch}, w, at::kBFloat16);
  FB_CALL(fb_conv_pack_filters, w.data_ptr<float>(), out.data_ptr(), s.O, s.C, s.kh, s.kw, s.sh, s.sw, s.eh, s.ew, pitch,
          dgrad, cur_stream());
  return out;
}

// x [B, C, H, W] fp32 as the operand z of the convolution.
Tensor packed_input(const Tensor& x, const Shape& s) {
  Tensor z = empty({s.B, s.Hz, s.Wz, s.Cz}, x, at::kBFloat16);
  FB_CALL(fb_conv_pack_input, x.data_ptr<float>(), nullptr, z.data_ptr(), s.B, s.C, s.H, s.W, s.sh, s.sw, s.eh, s.ew, s.lph,
          s.lpw, s.Hz, s.Wz, s.Cz, cur_stream());
  return z;
}
// The convolution of z into out [B, Ho, Wo, O]; beta: added to an fp32 one.
void forward_product(const Tensor& z, const Tensor& w, const Tensor& out, const float* bias, const Shape& s, int act, bool beta) {
  Tensor wk = packed_filters(w, s, false);
  FB_CALL(fb_conv_igemm_epilogue, z.data_ptr(), wk.data_ptr(), out.data_ptr(), bias, nullptr, s.B, s.Hz, s.Wz, s.Cz, s.O, s.k2h,
          s.k2w, s.gph, s.gpw, s.strided ? 1 : s.dh, s.strided ? 1 : s.dw, s.O, is_bf16(out), act, beta, status(), cur_stream());
}
// Gradient of z from gh [B, Ho, Wo, Op], dy convolved with the filters in reverse, channels exchanged: out [B, Hz, Wz, rows]
// fp32, or bf16 where mask (of the same layout) is above zero.
Tensor input_product(const Tensor& gh, const Tensor& w, const Shape& s, const Tensor& mask = Tensor()) {
  Tensor wt = packed_filters(w, s, true);
  const int rows = s.eh * s.ew * s.C, dh = s.strided ? 1 : s.dh, dw = s.strided ? 1 : s.dw;
  Tensor dz = empty({s.B, s.Hz, s.Wz, rows}, gh, mask.defined() ? at::kBFloat16 : at::kFloat);
  FB_CALL(fb_conv_igemm_epilogue, gh.data_ptr(), wt.data_ptr(), dz.data_ptr(), nullptr, ptr(mask), s.B, s.Ho, s.Wo, s.Op, rows,
          s.k2h, s.k2w, dh * (s.k2h - 1) - s.gph, dw * (s.k2w - 1) - s.gpw, dh, dw, rows, mask.defined(), FB_ACT_NONE, 0, status(),
          cur_stream());
  return dz;
}
// That of x, plus add (add_mask: where that is set; stride 1).
Tensor input_grad(const Tensor& gh, const Tensor& w, const Shape& s, const Tensor& add = Tensor(), const Tensor& add_mask = Tensor()) {
  Tensor dz = input_product(gh, w, s), dx = empty({s.B, s.C, s.H, s.W}, gh, at::kFloat);
  const int rows = s.eh * s.ew * s.C;
  if (s.strided)
    FB_CALL(fb_s2d_nhwc_to_nchw_add, dz.data_ptr<float>(), fptr(add), dx.data_ptr<float>(), s.B, s.C, s.H, s.W, s.sh, s.sw, s.eh,
            s.ew, s.ph, s.pw, s.Hz, s.Wz, rows, cur_stream());
  else
    FB_CALL(fb_nhwc_to_nchw_masks, dz.data_ptr<float>(), fptr(add), static_cast<const unsigned char*>(ptr(add_mask)),
            dx.data_ptr<float>(), nullptr, s.B, s.C, static_cast<ll>(s.H) * s.W, rows, 0, cur_stream());
  return dx;
}
Tensor filter_grad(const Tensor& gh, const Tensor& z, const Shape& s) {
  const int taps = s.k2h * s.k2w, dh = s.strided ? 1 : s.dh, dw = s.strided ? 1 : s.dw;
  const int splits = fb_conv_wgrad_splits(s.B, s.Ho, s.Wo, s.O, s.Cz, taps);
  Tensor part = empty({splits, s.O, taps, s.Cz}, gh, at::kFloat), dwt = empty({s.O, s.C, s.kh, s.kw}, gh, at::kFloat);
  FB_CALL(fb_conv_wgrad, gh.data_ptr(), z.data_ptr(), part.data_ptr<float>(), s.B, s.Hz, s.Wz, s.Cz, s.O, s.Op, s.k2h, s.k2w,
          s.gph, s.gpw, dh, dw, status(), cur_stream());
  FB_CALL(fb_conv_fold_wgrad, part.data_ptr<float>(), dwt.data_ptr<float>(), splits, s.O, s.C, s.kh, s.kw, s.sh, s.sw, s.eh, s.ew,
          s.Cz, cur_stream());
  return dwt;
}

struct ConvNode : Node {
  SavedVariable z_, w_, y_;
  Shape s;
  int act = 0;
  bool has_bias = false, has_add = false;
  at::ScalarType x_dtype = at::kFloat, add_dtype = at::kFloat;
  std::string name() const override { return "FerrumConvBackward"; }
  void release_variables() override {
    for (SavedVariable* v : {&z_, &w_, &y_}) v->reset_data();
  }
  variable_list apply(variable_list&& grads) override {
    variable_list out(4);  // x, w, bias, add
    if (!grads[0].defined()) return out;
    Tensor z = z_.unpack(), w = w_.unpack(), y = act != FB_ACT_NONE ? y_.unpack(shared_from_this()) : Tensor();
    NoAutograd below;
    w = f32c(w);
    z = contig(z);
    if (y.defined()) y = contig(y);
    Tensor g = f32c(grads[0]);
    if (has_add && task_should_compute_output(3)) out[3] = cast(g, add_dtype);
    // the gradient in front of the activation
    Tensor gh = empty({s.B, s.Ho, s.Wo, s.Op}, g, at::kBFloat16);
    FB_CALL(fb_conv_pack_input, g.data_ptr<float>(), fptr(y), gh.data_ptr(), s.B, s.O, s.Ho, s.Wo, 1, 1, 1, 1, 0, 0, s.Ho,
            s.Wo, s.Op, cur_stream());
    if (task_should_compute_output(0)) out[0] = cast(input_grad(gh, w, s), x_dtype);
    if (task_should_compute_output(1)) out[1] = filter_grad(gh, z, s);
    if (has_bias && task_should_compute_output(2)) {
      Tensor db = empty({s.Op}, g, at::kFloat);
      FB_CALL(fb_colsum, gh.data_ptr(), db.data_ptr<float>(), static_cast<ll>(s.B) * s.Ho * s.Wo, s.Op, FB_DT_BF16, 0,
              cur_stream());
      out[2] = db.slice(0, 0, s.O);
    }
    return out;
  }
};

Tensor conv2d(const Tensor& x, const Tensor& weight, const c10::optional<Tensor>& bias_,
              const c10::optional<Tensor>& add_, std::vector<int64_t> stride, std::vector<int64_t> padding,
              std::vector<int64_t> dilation, int act) {
  NoAutograd below;
  const Tensor bias = bias_.value_or(Tensor()), add = add_.value_or(Tensor());
  TORCH_CHECK_VALUE(x.dim() == 4 && weight.dim() == 4 && x.size(1) == weight.size(1),
                    "conv2d: [B, C, H, W] and [O, C, kh, kw] expected, got ", x.sizes(), " and ", weight.sizes());
  TORCH_CHECK_VALUE(stride.size() == 2 && padding.size() == 2 && dilation.size() == 2, "conv2d: pairs expected");
  // Negative padding is a crop; the space-to-depth kernels have none.
  TORCH_CHECK_VALUE(stride[0] > 0 && stride[1] > 0 && dilation[0] > 0 && dilation[1] > 0 &&
                        ((padding[0] >= 0 && padding[1] >= 0) || (stride[0] == 1 && stride[1] == 1)),
                    "conv2d: strides ", stride, ", padding ", padding, ", dilation ", dilation);
  TORCH_CHECK_VALUE(act == FB_ACT_NONE || act == FB_ACT_RELU, "conv2d: no epilogue evaluates activation ", act);
  TORCH_CHECK_VALUE(act == FB_ACT_NONE || !add_.has_value(), "conv2d: an added tensor or an activation, not both");
  check_on(x, weight, "the weight");
  if (bias.defined()) {
    check_on(x, bias, "the bias");
    TORCH_CHECK_VALUE(bias.numel() == weight.size(0), "conv2d: ", weight.size(0), " biases expected, got ", bias.numel());
  }
  Tensor xc = f32c(x), w = f32c(weight), b = bias.defined() ? f32c(bias) : bias;
  const Shape s = shape_of(xc.sizes(), w.sizes(), stride, padding, dilation);
  Tensor a;
  if (add.defined()) {
    check_on(x, add, "the added tensor");
    TORCH_CHECK_VALUE(add.sizes() == at::IntArrayRef({s.B, s.O, s.Ho, s.Wo}), "conv2d: an added tensor of the result's size ",
                      "expected, got ", add.sizes());
    a = f32c(add);
  }
  Tensor z = packed_input(xc, s), y = empty({s.B, s.O, s.Ho, s.Wo}, xc, at::kFloat);
  Tensor yh = empty({s.B, s.Ho, s.Wo, s.O}, xc, at::kFloat);
  forward_product(z, w, yh, fptr(b), s, FB_ACT_NONE, false);
  FB_CALL(fb_nhwc_to_nchw_f32, yh.data_ptr<float>(), fptr(a), y.data_ptr<float>(), s.B, s.O, static_cast<ll>(s.Ho) * s.Wo,
          s.O, act == FB_ACT_RELU, cur_stream());
  if (wants_grad({&x, &weight, &bias, &add})) {
    auto n = make_node<ConvNode>(x, weight, bias, add);
    n->s = s;
    n->act = act;
    n->has_bias = bias.defined();
    n->has_add = add.defined();
    n->x_dtype = x.scalar_type();
    if (add.defined()) n->add_dtype = add.scalar_type();
    n->z_ = below.keep(z);
    n->w_ = below.keep(weight);
    torch::autograd::set_history(y, n);
    if (act != FB_ACT_NONE) n->y_ = below.keep(y, true);
  }
  return y;
}

// ------------------------------------------------------------------------------------------- a residual block as one node
// relu(conv2(relu(conv1(x))) + identity), identity = x or a convolution of x; fp32 NCHW in and out.  Between the convolutions
// everything stays NHWC: the first product writes the bf16 operand of the second (the values that a layout pass would round to),
// its gradient comes back masked in bf16 the same way, the second product adds itself to the shortcut's, and the gradient behind
// the last ReLU is laid out once for both.  That ReLU's mask is kept as bytes of its own, so the result may be changed in place.
// 64 images, 64 -> 128 channels, 56 x 56, stride 2, a training step: 378 us as four nodes, 302 so.
struct BlockNode : Node {
  SavedVariable z1_, z2_, zd_, w1_, w2_, wd_, mask_;
  Shape s1, s2, sd;
  bool down = false;
  std::string name() const override { return "FerrumConvBlockBackward"; }
  void release_variables() override {
    for (SavedVariable* v : {&z1_, &z2_, &zd_, &w1_, &w2_, &wd_, &mask_}) v->reset_data();
  }
  variable_list apply(variable_list&& grads) override {
    variable_list out(4);  // x, w1, w2, wd
    if (!grads[0].defined()) return out;
    Tensor z1 = contig(z1_.unpack()), z2 = contig(z2_.unpack()), mask = contig(mask_.unpack());
    Tensor w1 = w1_.unpack(), w2 = w2_.unpack(), zd, wd;
    if (down) {
      zd = contig(zd_.unpack());
      wd = wd_.unpack();
    }
    NoAutograd below;
    w1 = f32c(w1);
    w2 = f32c(w2);
    if (down) wd = f32c(wd);
    const bool need_x = task_should_compute_output(0), need_1 = task_should_compute_output(1);
    Tensor dy = f32c(grads[0]), gh = empty({s2.B, s2.Ho, s2.Wo, s2.Op}, dy, at::kBFloat16);
    FB_CALL(fb_conv_pack_masked, dy.data_ptr<float>(), mask.data_ptr<uint8_t>(), gh.data_ptr(), s2.B, s2.O, s2.Ho, s2.Wo, s2.Op,
            cur_stream());
    if (task_should_compute_output(2)) out[2] = filter_grad(gh, z2, s2);
    if (down && task_should_compute_output(3)) out[3] = filter_grad(gh, zd, sd);
    Tensor dx;
    if (need_x || need_1) {
      Tensor g1 = input_product(gh, w2, s2, z2);
      if (need_1) out[1] = filter_grad(g1, z1, s1);
      if (need_x) dx = down ? input_grad(g1, w1, s1) : input_grad(g1, w1, s1, dy, mask);
    }
    if (need_x && down) dx = input_grad(gh, wd, sd, dx);
    out[0] = dx;
    return out;
  }
};

typedef std::vector<std::vector<int64_t>> Geometry;  // stride, padding, dilation

// Arguments as nn/conv.py (block_fused) lets them through: no biases, the channels between the convolutions in whole octets.
Tensor conv_block(const Tensor& x, const Tensor& w1, const Tensor& w2, const c10::optional<Tensor>& wd_, const Geometry& g1,
                  const Geometry& g2, const Geometry& gd) {
  NoAutograd below;
  const Tensor wd = wd_.value_or(Tensor());
  TORCH_CHECK_VALUE(x.dim() == 4 && w1.dim() == 4 && w2.dim() == 4 && x.size(1) == w1.size(1) && w1.size(0) == w2.size(1) &&
                        w1.size(0) % 8 == 0 && is_f32(x),
                    "conv_block: fp32 [B, C, H, W] and matching filters expected, got ", x.sizes(), ", ", w1.sizes(), ", ", w2.sizes());
  for (const Geometry* g : {&g1, &g2, &gd}) {
    if (g == &gd && !wd.defined()) continue;
    TORCH_CHECK_VALUE(g->size() == 3, "conv_block: stride, padding and dilation expected");
    for (const auto& v : *g) TORCH_CHECK_VALUE(v.size() == 2, "conv_block: pairs expected");
    const auto &st = (*g)[0], &pad = (*g)[1], &dil = (*g)[2];
    TORCH_CHECK_VALUE(st[0] > 0 && st[1] > 0 && dil[0] > 0 && dil[1] > 0 &&
                          ((pad[0] >= 0 && pad[1] >= 0) || (st[0] == 1 && st[1] == 1)),
                      "conv_block: strides ", st, ", padding ", pad, ", dilation ", dil);
  }
  check_on(x, w1, "a filter");
  check_on(x, w2, "a filter");
  Tensor xc = f32c(x), f1 = f32c(w1), f2 = f32c(w2), fd;
  const Shape s1 = shape_of(xc.sizes(), f1.sizes(), g1[0], g1[1], g1[2]);
  const Shape s2 = shape_of({s1.B, s1.O, s1.Ho, s1.Wo}, f2.sizes(), g2[0], g2[1], g2[2]);
  TORCH_CHECK_VALUE(!s2.strided && s1.Ho > 0 && s1.Wo > 0, "conv_block: the second convolution has a stride");
  Shape sd = s2;
  if (wd.defined()) {
    check_on(x, wd, "a filter");
    TORCH_CHECK_VALUE(wd.dim() == 4 && wd.size(1) == x.size(1), "conv_block: filters of the shortcut expected, got ", wd.sizes());
    fd = f32c(wd);
    sd = shape_of(xc.sizes(), fd.sizes(), gd[0], gd[1], gd[2]);
    TORCH_CHECK_VALUE(sd.O == s2.O && sd.Ho == s2.Ho && sd.Wo == s2.Wo, "conv_block: the shortcut's result has another size");
  } else {
    TORCH_CHECK_VALUE(!s1.strided && s1.C == s2.O && s1.H == s2.Ho && s1.W == s2.Wo, "conv_block: the result has another size than x");
  }
  Tensor z1 = packed_input(xc, s1), z2 = empty({s1.B, s1.Ho, s1.Wo, s1.O}, xc, at::kBFloat16), zd;
  forward_product(z1, f1, z2, nullptr, s1, FB_ACT_RELU, false);
  Tensor yh = empty({s2.B, s2.Ho, s2.Wo, s2.O}, xc, at::kFloat), y = empty({s2.B, s2.O, s2.Ho, s2.Wo}, xc, at::kFloat), mask;
  if (wd.defined()) {
    zd = packed_input(xc, sd);
    forward_product(zd, fd, yh, nullptr, sd, FB_ACT_NONE, false);
  }
  forward_product(z2, f2, yh, nullptr, s2, FB_ACT_NONE, wd.defined());
  const bool grad = wants_grad({&x, &w1, &w2, &wd});
  if (grad) mask = empty(y.sizes(), y, at::kByte);
  FB_CALL(fb_nhwc_to_nchw_masks, yh.data_ptr<float>(), wd.defined() ? nullptr : xc.data_ptr<float>(), nullptr, y.data_ptr<float>(),
          static_cast<unsigned char*>(ptr(mask)), s2.B, s2.O, static_cast<ll>(s2.Ho) * s2.Wo, s2.O, 1, cur_stream());
  if (grad) {
    auto n = make_node<BlockNode>(x, w1, w2, wd);
    n->s1 = s1;
    n->s2 = s2;
    n->sd = sd;
    n->down = wd.defined();
    n->z1_ = below.keep(z1);
    n->z2_ = below.keep(z2);
    n->zd_ = below.keep(zd);
    n->w1_ = below.keep(w1);
    n->w2_ = below.keep(w2);
    n->wd_ = below.keep(wd);
    n->mask_ = below.keep(mask);
    torch::autograd::set_history(y, n);
  }
  return y;
}

}  // namespace

void bind_conv(py::module_& m) {
  m.def("conv2d", &conv2d);
  m.def("conv_block", &conv_block);
}

}  // namespace fbn
