// Embedding lookups and blockwise attention.
#include "native.h"

#include <ATen/cuda/cub.h>

namespace fbn {
namespace {

struct EmbeddingNode : Node {
  SavedVariable idx_;
  int64_t vocab = 0, dim = 0, group = 1;
  ll padding = -1;
  std::shared_ptr<Sink> sink;
  std::string name() const override { return "FerrumEmbeddingBackward"; }
  void release_variables() override { idx_.reset_data(); }
  variable_list apply(variable_list&& grads) override {
    variable_list out(1);
    if (!grads[0].defined()) return out;
    Tensor idx = idx_.unpack(), dw, sorted, perm, g2;
    const int64_t n = idx.numel(), pitch = (n + 127) / 128 * 128;
    // Pairs of 32 bits, sorted by the bits that a row number has (two passes of the radix sort for a table of 50000 rows, where
    // at::sort makes four, and positions and copies of its own): 131072 indices 57 -> 27 us with the gaps between the launches.
    const bool pairs = vocab < 0x7fffffff && n < 0x7fffffff;
    {
      NoAutograd below;
      g2 = contig(grads[0]).reshape({-1, dim});
      if (pairs && n > 0) {
        int bits = 1;
        while (vocab >> bits) ++bits;
        sorted = empty({4, pitch}, idx, at::kInt);
        int32_t* at = sorted.data_ptr<int32_t>();
        FB_CALL(fb_embedding_pairs, reinterpret_cast<const ll*>(contig(idx).data_ptr<int64_t>()), at + 2 * pitch, at + 3 * pitch,
                n, vocab, group, cur_stream());
        at::cuda::cub::radix_sort_pairs(at + 2 * pitch, at, at + 3 * pitch, at + pitch, n, false, 0, bits);
      } else if (!pairs) {
        std::tie(sorted, perm) = at::sort(idx.reshape({-1}), /*stable=*/true, /*dim=*/0, /*descending=*/false);
      }
    }
    bool add = false;
    if (sink) {  // accumulate straight into the data-parallel gradient arena
      py::gil_scoped_acquire gil;
      py::tuple r = py::handle(sink->sink).attr("acquire")(py::handle(sink->param));
      dw = r[0].cast<Tensor>();
      add = r[1].cast<bool>();
      if (!add) dw.zero_();
    } else {
      dw = at::zeros({vocab, dim}, g2.options().dtype(at::kFloat));
    }
    const float scale = 1.f / static_cast<float>(group);
    if (!pairs)
      FB_CALL(fb_embedding_bwd_sorted, g2.data_ptr(), reinterpret_cast<const ll*>(sorted.data_ptr<int64_t>()),
              reinterpret_cast<const ll*>(perm.data_ptr<int64_t>()), dw.data_ptr<float>(), n, static_cast<int>(dim),
              static_cast<int>(group), scale, padding, vocab, dt(g2), cur_stream());
    else if (n > 0) {
      const auto scatter = add ? fb_embedding_bwd_pairs : fb_embedding_bwd_pairs_zeroed;
      FB_CALL(scatter, g2.data_ptr(), sorted.data_ptr<int32_t>(), sorted.data_ptr<int32_t>() + pitch, dw.data_ptr<float>(), n,
              static_cast<int>(dim), static_cast<int>(group), scale, padding, vocab, dt(g2), cur_stream());
    }
    if (sink) sink_ready(*sink);
    else out[0] = dw;
    return out;
  }
};

Tensor embedding(const Tensor& weight, const Tensor& idx_, ll padding, bool pool, bool out_bf16, py::object sink) {
  NoAutograd below;
  TORCH_CHECK_VALUE(weight.dim() == 2 && (!pool || idx_.dim() == 2), "embedding: a table of two dimensions expected, got ",
                    weight.sizes(), " and indices ", idx_.sizes());
  if (idx_.numel() > 0) check_on(weight, idx_, "the index tensor");
  Tensor w = contig(weight), idx = contig(idx_);
  const int64_t V = w.size(0), D = w.size(1);
  const auto st = out_bf16 ? at::kBFloat16 : at::kFloat;
  Tensor y;
  if (pool) {
    y = empty({idx.size(0), D}, w, st);
    FB_CALL(fb_embedding_meanpool_fwd, w.data_ptr<float>(), reinterpret_cast<const ll*>(idx.data_ptr<int64_t>()),
            y.data_ptr(), idx.size(0), static_cast<int>(idx.size(1)), static_cast<int>(D), V, dt(y), cur_stream());
  } else {
    std::vector<int64_t> sizes(idx.sizes().begin(), idx.sizes().end());
    sizes.push_back(D);
    y = empty(sizes, w, st);
    FB_CALL(fb_embedding_fwd, w.data_ptr<float>(), reinterpret_cast<const ll*>(idx.data_ptr<int64_t>()), y.data_ptr(),
            idx.numel(), static_cast<int>(D), V, padding, dt(y), status(), cur_stream());
  }
  if (wants_grad({&weight})) {
    auto n = make_node<EmbeddingNode>(weight);
    n->idx_ = below.keep(idx);
    n->vocab = V;
    n->dim = D;
    n->group = pool ? idx.size(1) : 1;
    n->padding = padding;
    n->sink = make_sink(sink, py::cast(weight));
    torch::autograd::set_history(y, n);
  }
  return y;
}

// ------------------------------------------------------------------------------------ recurrent sequences
// One LSTM (gates = 4) or GRU (gates = 3) layer over proj [T, B, gates H]; returns hs [T, B, H] and, for LSTM, the
// last cell state [B, H].  The recurrence runs in one launch per direction; the weight gradient of all steps is one
// product over T B rows.
struct RnnSeqNode : Node {
  SavedVariable w_, h0_, c0_, hs_, cs_, saved_;
  int gates = 4;
  bool has_bias = false;
  std::string name() const override { return "FerrumRnnSeqBackward"; }
  void release_variables() override {
    for (SavedVariable* s : {&w_, &h0_, &c0_, &hs_, &cs_, &saved_}) s->reset_data();
  }
  variable_list apply(variable_list&& grads) override {
    variable_list out(5);  // proj, w, bias, h0, c0
    Tensor w = w_.unpack(), h0 = h0_.unpack(), c0 = c0_.unpack(), hs = hs_.unpack(), cs = cs_.unpack(),
           saved = saved_.unpack();
    NoAutograd below;
    w = contig(w);
    if (h0.defined()) h0 = f32c(h0);
    if (c0.defined()) c0 = f32c(c0);
    Tensor dhs = grads[0].defined() ? f32c(grads[0]) : Tensor();
    Tensor dc = grads.size() > 1 && grads[1].defined() ? f32c(grads[1]) : Tensor();
    if (!dhs.defined() && !dc.defined()) return out;
    const int64_t T = hs.size(0), B = hs.size(1), H = hs.size(2), GH = gates * H;
    Tensor dxi = empty({T, B, GH}, hs, at::kFloat), dhh = gates == 3 ? empty({T, B, GH}, hs, at::kFloat) : dxi;
    Tensor dh0 = task_should_compute_output(3) ? empty({B, H}, hs, at::kFloat) : Tensor();
    Tensor dc0 = gates == 4 && task_should_compute_output(4) ? empty({B, H}, hs, at::kFloat) : Tensor();
    FB_CALL(fb_rnn_seq_bwd, gates, w.data_ptr<float>(), fptr(h0), fptr(c0), hs.data_ptr<float>(), fptr(cs),
            saved.data_ptr<float>(), fptr(dhs), fptr(dc), dxi.data_ptr<float>(),
            gates == 3 ? dhh.data_ptr<float>() : nullptr, fptr_mut(dh0), fptr_mut(dc0), static_cast<int>(T),
            static_cast<int>(B), static_cast<int>(H), status(), cur_stream());
    out[0] = dxi;
    if (task_should_compute_output(1)) {
      Tensor dw = empty({GH, H}, hs, at::kFloat);
      const float* d = dhh.data_ptr<float>();
      const bool first = h0.defined();  // the step from a zero state contributes nothing
      if (T > 1)
        gemm(Op{d + B * GH, GH, (T - 1) * B, 1, GH, false}, Op{hs.data_ptr(), H, (T - 1) * B, 1, H, false}, nullptr, 0,
             dw.data_ptr(), H, false);
      if (first)
        gemm(Op{d, GH, B, 1, GH, false}, Op{h0.data_ptr(), H, B, 1, H, false}, nullptr, 0, dw.data_ptr(), H, false,
             T > 1);
      if (T == 1 && !first) dw.zero_();
      out[1] = dw;
    }
    if (has_bias && task_should_compute_output(2)) {
      Tensor db = empty({GH}, hs, at::kFloat);
      FB_CALL(fb_colsum, dhh.data_ptr(), db.data_ptr<float>(), T * B, GH, FB_DT_F32, 0, cur_stream());
      out[2] = db;
    }
    out[3] = dh0;
    out[4] = dc0;
    return out;
  }
};

std::vector<Tensor> rnn_seq(int gates, const Tensor& proj, const Tensor& w, const c10::optional<Tensor>& bias_,
                            const c10::optional<Tensor>& h0_, const c10::optional<Tensor>& c0_) {
  NoAutograd below;
  const Tensor bias = bias_.value_or(Tensor()), h0 = h0_.value_or(Tensor()), c0 = c0_.value_or(Tensor());
  TORCH_CHECK_VALUE(proj.dim() == 3 && w.dim() == 2, "rnn_seq: [T, B, gates H] and [gates H, H] expected, got ",
                    proj.sizes(), " and ", w.sizes());
  const int64_t T = proj.size(0), B = proj.size(1), H = w.size(1), GH = gates * H;
  TORCH_CHECK_VALUE(proj.size(2) == GH && w.size(0) == GH, "rnn_seq: sizes do not match: ", proj.sizes(), " and ", w.sizes());
  TORCH_CHECK_VALUE(!bias.defined() || bias.sizes() == at::IntArrayRef({GH}), "rnn_seq: bias of [", GH, "] expected, got ",
                    bias.sizes());
  for (const Tensor* s : {&h0, &c0})
    TORCH_CHECK_VALUE(!s->defined() || s->sizes() == at::IntArrayRef({B, H}), "rnn_seq: initial state of [", B, ", ", H,
                      "] expected, got ", s->sizes());
  check_on(proj, w, "the recurrent matrix");
  if (bias.defined()) check_on(proj, bias, "the bias");
  if (h0.defined()) check_on(proj, h0, "the initial hidden state");
  if (c0.defined()) check_on(proj, c0, "the initial cell state");
  TORCH_CHECK_VALUE(proj.is_cuda(), "rnn_seq: a CUDA input expected");
  Tensor x = f32c(proj), wc = contig(w);
  Tensor b = bias.defined() ? contig(bias) : bias, h = h0.defined() ? f32c(h0) : h0, c = c0.defined() ? f32c(c0) : c0;
  const bool grad = wants_grad({&proj, &w, &bias, &h0, &c0});
  Tensor wt = empty({H, GH}, x, at::kFloat), hs = empty({T, B, H}, x, at::kFloat);
  // what the backward pass reads of the outputs is kept apart from them: a caller may change those in place
  Tensor kept = grad ? empty({T, B, H}, x, at::kFloat) : Tensor();
  Tensor cs = gates == 4 && grad ? empty({T, B, H}, x, at::kFloat) : Tensor();
  Tensor saved = grad ? empty({T, B, 4 * H}, x, at::kFloat) : Tensor();
  Tensor c_last = gates == 4 ? empty({B, H}, x, at::kFloat) : Tensor();
  FB_CALL(fb_transpose_2d, wc.data_ptr(), wt.data_ptr(), static_cast<int>(GH), static_cast<int>(H), 4, cur_stream());
  FB_CALL(fb_rnn_seq_fwd, gates, x.data_ptr<float>(), wt.data_ptr<float>(), fptr(b), fptr(h), fptr(c),
          hs.data_ptr<float>(), fptr_mut(kept), fptr_mut(cs), fptr_mut(saved), fptr_mut(c_last), static_cast<int>(T),
          static_cast<int>(B), static_cast<int>(H), status(), cur_stream());
  std::vector<Tensor> out{hs};
  if (gates == 4) out.push_back(c_last);
  if (grad) {
    auto n = make_node<RnnSeqNode>(proj, w, bias, h0, c0);
    n->gates = gates;
    n->has_bias = bias.defined();
    n->w_ = below.keep(w);
    n->h0_ = below.keep(h0);
    n->c0_ = below.keep(c0);
    n->cs_ = below.keep(cs);
    n->saved_ = below.keep(saved);
    n->hs_ = below.keep(kept);
    torch::autograd::set_history(out, n);
  }
  return out;
}

}  // namespace

void bind_layers(py::module_& m) {
  m.def("embedding", &embedding);
  m.def("rnn_seq", &rnn_seq);
  m.def("rnn_seq_supported", [](int gates, int batch, int hidden) { return fb_rnn_seq_supported(gates, batch, hidden) != 0; });
  m.def("rnn_seq_plan", &fb_rnn_seq_plan);
}

}  // namespace fbn
