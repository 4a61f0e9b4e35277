// Embedding lookups and blockwise attention.
#include "native.h"

namespace fbn {
namespace {

struct EmbeddingNode : Node {
  Tensor idx;
  int64_t vocab = 0, dim = 0, group = 1;
  ll padding = -1;
  std::shared_ptr<Sink> sink;
  std::string name() const override { return "FerrumEmbeddingBackward"; }
  void release_variables() override { idx = Tensor(); }
  variable_list apply(variable_list&& grads) override {
    variable_list out(1);
    if (!grads[0].defined()) return out;
    TORCH_CHECK(idx.defined(), "Trying to backward through the graph a second time");
    Tensor dw, sorted, perm, g2;
    {
      NoAutograd below;
      g2 = contig(grads[0]).reshape({-1, dim});
      std::tie(sorted, perm) = at::sort(idx.reshape({-1}), /*stable=*/true, /*dim=*/0, /*descending=*/false);
    }
    if (sink) {  // accumulate straight into the data-parallel gradient arena
      py::gil_scoped_acquire gil;
      py::tuple r = py::handle(sink->sink).attr("acquire")(py::handle(sink->param));
      dw = r[0].cast<Tensor>();
      if (!r[1].cast<bool>()) dw.zero_();
    } else {
      dw = at::zeros({vocab, dim}, g2.options().dtype(at::kFloat));
    }
    FB_CALL(fb_embedding_bwd_sorted, g2.data_ptr(), reinterpret_cast<const ll*>(sorted.data_ptr<int64_t>()),
            reinterpret_cast<const ll*>(perm.data_ptr<int64_t>()), dw.data_ptr<float>(), sorted.numel(),
            static_cast<int>(dim), static_cast<int>(group), 1.f / static_cast<float>(group), padding, vocab, dt(g2),
            cur_stream());
    if (sink) sink_ready(*sink);
    else out[0] = dw;
    return out;
  }
};

Tensor embedding(const Tensor& weight, const Tensor& idx_, ll padding, bool pool, bool out_bf16, py::object sink) {
  NoAutograd below;
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
    n->idx = idx;
    n->vocab = V;
    n->dim = D;
    n->group = pool ? idx.size(1) : 1;
    n->padding = padding;
    n->sink = make_sink(sink, py::cast(weight));
    torch::autograd::set_history(y, n);
  }
  return y;
}

}  // namespace

void bind_layers(py::module_& m) { m.def("embedding", &embedding); }

}  // namespace fbn
