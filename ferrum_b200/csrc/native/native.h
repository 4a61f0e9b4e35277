// Host path of the differentiable ops: autograd nodes and launch code in C++, reached from Python through one call
// per op.  The kernels stay behind the C interface of include/ferrum_kernels.h; their symbols come from the kernel
// library that the Python side has loaded globally before this module (so the index-checking build works too).
#pragma once
#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <torch/csrc/autograd/forward_grad.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/variable.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/utils/pybind.h>

#include <atomic>
#include <memory>

#include "../include/ferrum_kernels.h"

namespace fbn {

using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;
typedef long long ll;

// ---------------------------------------------------------------------------------------------- launches
extern std::atomic<ll> g_launches;     // kernel launchers called so far
extern std::atomic<bool> g_profiling;  // record two events around each launcher
void profile_begin(const char* name);
void profile_end();
[[noreturn]] void launch_failed(const char* name, int rc);

template <class Fn>
inline void launch(const char* name, Fn&& fn) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  const bool prof = g_profiling.load(std::memory_order_relaxed);
  if (prof) profile_begin(name);
  const int rc = fn();
  if (prof) profile_end();
  if (rc != 0) launch_failed(name, rc);
}
#define FB_CALL(fn, ...) ::fbn::launch(#fn, [&] { return fn(__VA_ARGS__); })

inline cudaStream_t cur_stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
int32_t* status();  // host-mapped status block of the current device

// ------------------------------------------------------------------------------------------- tensor helpers
inline bool is_bf16(const Tensor& t) { return t.scalar_type() == at::kBFloat16; }
inline bool is_f32(const Tensor& t) { return t.scalar_type() == at::kFloat; }
inline int dt(const Tensor& t) {
  if (is_f32(t)) return FB_DT_F32;
  if (is_bf16(t)) return FB_DT_BF16;
  TORCH_CHECK_TYPE(false, "kernel supports fp32 / bf16, got ", t.scalar_type());
}
inline Tensor empty(at::IntArrayRef sizes, const Tensor& like, at::ScalarType st) {
  return at::empty(sizes, like.options().dtype(st).requires_grad(false).memory_format(at::MemoryFormat::Contiguous));
}
inline Tensor contig(const Tensor& t) { return t.is_contiguous() ? t : t.contiguous(); }
inline const float* fptr(const Tensor& t) { return t.defined() ? t.data_ptr<float>() : nullptr; }
inline float* fptr_mut(const Tensor& t) { return t.defined() ? t.data_ptr<float>() : nullptr; }
inline void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
inline ll rows_of(const Tensor& t) {
  const ll c = t.dim() ? t.size(-1) : 1;
  return c > 0 ? t.numel() / c : 0;
}
Tensor cast(const Tensor& t, at::ScalarType st);  // the cast kernel for fp32 <-> bf16, contiguous result
inline Tensor f32c(const Tensor& t) { return contig(is_f32(t) ? t : cast(t, at::kFloat)); }
// The kernels get bare pointers: what they read must be on the input's device and of the size they go by.
inline void check_on(const Tensor& input, const Tensor& t, const char* what) {
  TORCH_CHECK_VALUE(t.device() == input.device(), what, " is on ", t.device(), ", the input on ", input.device());
}
// A bias or a scale: a value for each of the n columns.
inline void check_columns(const Tensor& input, const Tensor& t, int64_t n, const char* what) {
  if (!t.defined()) return;
  check_on(input, t, what);
  TORCH_CHECK_VALUE(t.numel() == n, what, " has ", t.numel(), " values, expected ", n);
}
inline Tensor as2d(const Tensor& t) { return t.dim() == 2 ? t : t.reshape({-1, t.size(-1)}); }

// ------------------------------------------------------------------------------------------------ autograd
// The ops run below the autograd keys: a tangent would be lost there without a word.
inline void refuse_tangents(std::initializer_list<const Tensor*> ts) {
  if (!torch::autograd::ForwardADLevel::try_get_by_idx(0)) return;  // nobody is in a dual level
  for (const Tensor* t : ts)
    TORCH_CHECK_NOT_IMPLEMENTED(!t->defined() || !t->_fw_grad(/*level=*/0).defined(),
                                "this op has no forward-mode derivative (a dual tensor was given)");
}
inline bool wants_grad(std::initializer_list<const Tensor*> ts) {
  refuse_tangents(ts);
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor* t : ts)
    if (t->defined() && t->requires_grad()) return true;
  return false;
}
template <class N, class... T>
inline std::shared_ptr<N> make_node(const T&... inputs) {
  std::shared_ptr<N> n(new N(), torch::autograd::deleteNode);
  n->set_next_edges(torch::autograd::collect_next_edges(inputs...));
  return n;
}
// Inside an op and inside a node's apply: the tensor methods used there record nothing of their own.
struct NoAutograd {
  const c10::impl::LocalDispatchKeySet outer = c10::impl::tls_local_dispatch_key_set();
  at::AutoDispatchBelowADInplaceOrView guard;
  // A tensor that the backward pass reads.  Saved-tensor hooks are the user's code (the recomputation of a checkpoint
  // among them): they run with the dispatch state of the op's caller, and an apply unpacks before it sets its guard.
  SavedVariable keep(const Tensor& t, bool is_output = false) const {
    if (!t.defined()) return SavedVariable();
    c10::impl::ForceDispatchKeyGuard user(outer);
    try {
      return SavedVariable(t, is_output);
    } catch (python_error& e) {  // raised by a hook, by way of pybind
      e.restore();
      throw py::error_already_set();
    }
  }
};

Tensor add(const Tensor& a, const Tensor& b);
Tensor unary(const Tensor& x, int op, double alpha, double beta);

// ---------------------------------------------------------------------------------------------------- GEMM
// A GEMM operand as an [rows, K] view given by element strides.
struct Op {
  const void* p;
  ll rows, k, s_row, s_k;
  bool bf16;
  Op t() const { return Op{p, k, rows, s_k, s_row, bf16}; }
};
inline Op op2d(const Tensor& t) { return Op{t.data_ptr(), t.size(0), t.size(1), t.stride(0), t.stride(1), is_bf16(t)}; }
extern std::atomic<bool> g_tf32, g_use_2cta;
extern std::atomic<int> g_max_ctas;
bool tma_ok(const Op& a);
// out[M, N] (row pitch ldc) = act(a b^T + bias), += out when `accumulate`; act_grad: see fb_gemm_bf16.  `splits`: bf16
// products of few output tiles may divide K over a cluster.  Set for weight gradients alone: forward results and input
// gradients of aligned bf16 operands keep one order of summation, so that a row's result depends neither on the rows
// beside it nor on whether gradients are recorded (carried through eight bf16 layers, another order moved the logits by
// 0.9 %, as far from the exact ones as before).
void gemm(const Op& a, const Op& b, const float* bias, int act, void* out, ll ldc, bool out_bf16,
          bool accumulate = false, void* act_grad = nullptr, const Tensor* like = nullptr, bool tf32 = false, bool splits = false);

// --------------------------------------------------------------------------------------------------- sinks
// Where the data-parallel engine wants a weight gradient (Python object with acquire / ready / try_push).
struct Sink {
  PyObject* sink = nullptr;
  PyObject* param = nullptr;
  ~Sink();
};
std::shared_ptr<Sink> make_sink(py::handle sink, py::handle param);
// dW = g^T x ([N, K], fp32): into the sink's buffer, or pushed to the shard owners by the GEMM's epilogue.
void wgrad_to_sink(Sink& s, const Tensor& g2, const Tensor& x2);
void sink_ready(Sink& s);

void bind_linear(py::module_& m);
void bind_elementwise(py::module_& m);
void bind_layers(py::module_& m);
void bind_conv(py::module_& m);
void bind_optim(py::module_& m);

}  // namespace fbn
