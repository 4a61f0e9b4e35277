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
    if (task_should_compute_output(0)) {  // dy convolved with the filters in reverse, channels exchanged
      Tensor wt = packed_filters(w, s, true);
      const int rows = s.eh * s.ew * s.C, dh = s.strided ? 1 : s.dh, dw = s.strided ? 1 : s.dw;
      Tensor dx = empty({s.B, s.C, s.H, s.W}, g, at::kFloat), dz = empty({s.B, s.Hz, s.Wz, rows}, g, at::kFloat);
      FB_CALL(fb_conv_igemm, gh.data_ptr(), wt.data_ptr(), dz.data_ptr(), nullptr, s.B, s.Ho, s.Wo, s.Op, rows, s.k2h, s.k2w,
              dh * (s.k2h - 1) - s.gph, dw * (s.k2w - 1) - s.gpw, dh, dw, rows, 0, status(), cur_stream());
      if (s.strided)
        FB_CALL(fb_s2d_nhwc_to_nchw_f32, dz.data_ptr<float>(), dx.data_ptr<float>(), s.B, s.C, s.H, s.W, s.sh, s.sw, s.eh,
                s.ew, s.ph, s.pw, s.Hz, s.Wz, rows, cur_stream());
      else
        FB_CALL(fb_nhwc_to_nchw_f32, dz.data_ptr<float>(), nullptr, dx.data_ptr<float>(), s.B, s.C,
                static_cast<ll>(s.H) * s.W, rows, 0, cur_stream());
      out[0] = cast(dx, x_dtype);
    }
    if (task_should_compute_output(1)) {
      const int taps = s.k2h * s.k2w, dh = s.strided ? 1 : s.dh, dw = s.strided ? 1 : s.dw;
      const int splits = fb_conv_wgrad_splits(s.B, s.Ho, s.Wo, s.O, s.Cz, taps);
      Tensor part = empty({splits, s.O, taps, s.Cz}, g, at::kFloat), dwt = empty({s.O, s.C, s.kh, s.kw}, g, at::kFloat);
      FB_CALL(fb_conv_wgrad, gh.data_ptr(), z.data_ptr(), part.data_ptr<float>(), s.B, s.Hz, s.Wz, s.Cz, s.O, s.Op, s.k2h,
              s.k2w, s.gph, s.gpw, dh, dw, status(), cur_stream());
      FB_CALL(fb_conv_fold_wgrad, part.data_ptr<float>(), dwt.data_ptr<float>(), splits, s.O, s.C, s.kh, s.kw, s.sh, s.sw,
              s.eh, s.ew, s.Cz, cur_stream());
      out[1] = dwt;
    }
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
  Tensor z = empty({s.B, s.Hz, s.Wz, s.Cz}, xc, at::kBFloat16), y = empty({s.B, s.O, s.Ho, s.Wo}, xc, at::kFloat);
  FB_CALL(fb_conv_pack_input, xc.data_ptr<float>(), nullptr, z.data_ptr(), s.B, s.C, s.H, s.W, s.sh, s.sw, s.eh, s.ew, s.lph,
          s.lpw, s.Hz, s.Wz, s.Cz, cur_stream());
  Tensor wk = packed_filters(w, s, false), yh = empty({s.B, s.Ho, s.Wo, s.O}, xc, at::kFloat);
  FB_CALL(fb_conv_igemm, z.data_ptr(), wk.data_ptr(), yh.data_ptr(), fptr(b), s.B, s.Hz, s.Wz, s.Cz, s.O, s.k2h, s.k2w, s.gph,
          s.gpw, s.strided ? 1 : s.dh, s.strided ? 1 : s.dw, s.O, 0, status(), cur_stream());
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

}  // namespace

void bind_conv(py::module_& m) { m.def("conv2d", &conv2d); }

}  // namespace fbn
