// Launch accounting, the GEMM dispatch and the module itself.
#include "native.h"

#include <c10/cuda/CUDAFunctions.h>
#include <mutex>
#include <vector>

extern "C" {
int32_t* fb_rt_status_ptr(void);
const char* fb_rt_error_string(int);
void* fb_rt_event_create(int timing);
int fb_rt_event_record(void* event, void* stream);
int fb_rt_event_synchronize(void* event);
int fb_rt_event_destroy(void* event);
float fb_rt_event_elapsed_ms(void* start, void* stop);
}

namespace fbn {

std::atomic<ll> g_launches{0};
std::atomic<bool> g_profiling{false};
std::atomic<bool> g_tf32{false}, g_use_2cta{true};
std::atomic<int> g_max_ctas{0};

// ------------------------------------------------------------------------------------------------ launches
struct Record {
  const char* name;
  void *e0, *e1;
};
static std::mutex g_prof_mutex;
static std::vector<Record> g_records;
static thread_local Record t_record;

void profile_begin(const char* name) {
  t_record.name = name;
  t_record.e0 = fb_rt_event_create(1);
  t_record.e1 = fb_rt_event_create(1);
  fb_rt_event_record(t_record.e0, cur_stream());
}
void profile_end() {
  fb_rt_event_record(t_record.e1, cur_stream());
  std::lock_guard<std::mutex> lock(g_prof_mutex);
  g_records.push_back(t_record);
}

void launch_failed(const char* name, int rc) {
  TORCH_CHECK(rc < 0, name, ": CUDA error ", rc, ": ", fb_rt_error_string(rc));
  TORCH_CHECK_VALUE(false, name, ": invalid argument (code ", rc, ")");
}

int32_t* status() {
  static std::atomic<int32_t*> ptrs[64];
  const int dev = c10::cuda::current_device();
  std::atomic<int32_t*>& slot = ptrs[dev & 63];
  int32_t* p = slot.load(std::memory_order_acquire);
  if (p == nullptr) {
    p = fb_rt_status_ptr();
    TORCH_CHECK(p != nullptr, "could not allocate the device status block");
    fb_layernorm_set_status(p);  // kernels without a status argument report here (one device per process)
    slot.store(p, std::memory_order_release);
  }
  return p;
}

Tensor cast(const Tensor& t, at::ScalarType st) {
  if (t.scalar_type() == st) return t;
  if (!((is_f32(t) && st == at::kBFloat16) || (is_bf16(t) && st == at::kFloat))) return t.to(st);
  Tensor x = contig(t), y = empty(x.sizes(), x, st);
  FB_CALL(fb_cast, x.data_ptr(), y.data_ptr(), x.numel(), dt(x), dt(y), cur_stream());
  return y;
}

// ---------------------------------------------------------------------------------------------------- GEMM
bool tma_ok(const Op& a) {
  const ll unit = a.bf16 ? 8 : 4;  // elements per 16 bytes
  if (reinterpret_cast<uintptr_t>(a.p) % 16) return false;
  if (a.s_k == 1) return a.s_row % unit == 0 && a.s_row >= a.k;
  if (a.s_row == 1) return a.s_k % unit == 0 && a.s_k >= a.rows;
  return false;
}

// bf16 operands that no TMA map describes, copied to a row pitch (or column pitch, whichever direction is contiguous)
// that one does describe; both in one launch.
static void aligned_copies(Op& a, Op& b, const at::TensorOptions& opt, Tensor& keep_a, Tensor& keep_b) {
  struct Copy {
    const void* src = nullptr;
    void* dst = nullptr;
    ll rows = 0, pitch = 0;
    int cols = 0;
  } c[2];
  int n = 0;
  for (int i = 0; i < 2; ++i) {
    Op& o = i ? b : a;
    if (tma_ok(o)) continue;
    Tensor& keep = i ? keep_b : keep_a;
    const bool mn = o.s_k != 1 && o.s_row == 1;
    const ll rows = mn ? o.k : o.rows, cols = mn ? o.rows : o.k, pitch = mn ? o.s_k : o.s_row, to = (cols + 7) / 8 * 8;
    keep = at::empty({rows, to}, opt);
    if ((mn || o.s_k == 1) && pitch >= cols) {
      c[n++] = Copy{o.p, keep.data_ptr(), rows, pitch, static_cast<int>(cols)};
    } else {  // neither direction is contiguous, or rows share elements
      keep.narrow(1, 0, cols).copy_(
          at::from_blob(const_cast<void*>(o.p), {rows, cols}, {mn ? o.s_k : o.s_row, mn ? o.s_row : o.s_k}, opt));
    }
    o = Op{keep.data_ptr(), o.rows, o.k, mn ? 1 : to, mn ? to : 1, true};
  }
  if (n > 0)
    FB_CALL(fb_repack_rows, c[0].src, c[0].dst, c[0].rows, c[0].cols, c[0].pitch, c[1].src, c[1].dst, c[1].rows, c[1].cols,
            c[1].pitch, cur_stream());
}
// Where results of any type take the copies (fp32 ones, weight gradients, only here).  The kernel that reads such operands
// in place adds its k-blocks in registers, rounded to nearest, the aligned kernels in one chain that truncates; an fp32
// result shows it, and where the copies gain little the exact kernel stays.  The line charges it 70 products
// (multiply-adds) per ns and a copy 6 us and 1.6 TB/s, though one launch of 4 us and 4 TB/s makes both copies; reductions
// that are no multiple of 8 stay in place altogether.  Weight gradients [N, K] of M rows, in place / copies + product in us
// (relative errors): M 777, 1001 x 1001 21.4 / 18.6 (9e-8 / 7e-7); 1024, 1001 x 1001 22.7 / 20.8 (9e-8 / 1e-6); 1024, 2049 x
// 2049 74 / 33; 4096, 1001 x 1001 62 / 32; 8192, 37 x 4095 62 / 56; 8192, 4095 x 4095 1526 / 311 (2e-7 / 9e-6).  With a
// single operand to copy and rows that the TMA unit can store the aligned kernels also save 3 us per million elements of
// the result: 64, 1001 x 2048 12.4 / 12.3; 512, 333 x 1024 13.0 / 16.4; 512, 1001 x 4096 45 / 16; 4096, 1001 x 1024 62 / 27.
static bool copies_repay(const Op& a, const Op& b, bool rows_tma) {
  if (a.k % 8 != 0) return false;
  double us = static_cast<double>(a.rows) * b.rows * a.k / 7e7, cost = 0.;
  int copies = 0;
  bool rows_first = true;  // the copied operands have their rows contiguous, as in a weight gradient
  for (const Op* o : {&a, &b})
    if (!tma_ok(*o)) {
      cost += 6. + static_cast<double>(o->rows) * o->k * 4 / 1.6e6;
      rows_first &= o->s_row == 1;
      ++copies;
    }
  if (copies != 1 || !rows_first || !rows_tma) return us > cost + 5.;
  us += static_cast<double>(a.rows) * b.rows * 3e-6;
  return us > cost - 2.;
}

// The same for products with a bf16 result (layers and gradients of activations) of any reduction: the rounding of the
// result (1.66e-3 of its norm either way; 1 in 500 to 2000 elements falls to the other neighbour) hides the difference,
// 1e-7 against 1e-6 at K = 1001 and 4e-6 at K = 4095.  A row's bits may change when the rows beside it pass this line
// (those of aligned operands never do).  In place against copy + product, us: 1024 x 1001 x 1001 19.1 / 3.7 + 13.8, 2048 x
// 1001 x 1001 30.3 / 4.6 + 14.0, 777 x 2049 x 2049 49.2 / 6.3 + 20.4, 512 x 4095 x 4095 84.9 / 16.6 + 32.0, 8191 x 4095 x
// 4095 1146 / 48 + 200; below 512 rows, without the pairs, 300 x 1001 x 4095 27.1 / 6.3 + 55.2.  (Both sides have become 5 - 15 %
// faster since.)
static bool repack_repays(const Op& a, const Op& b) {
  if (a.rows < 512 || b.rows < 128) return false;
  double cost = 14.;
  for (const Op* o : {&a, &b})
    if (!tma_ok(*o)) cost += static_cast<double>(o->rows) * o->k * 4 / 4e6;
  return static_cast<double>(a.rows) * b.rows * a.k / 7e7 > cost;
}

// fp32 products with a reduction this short do not repay the tensor-core kernel's set-up (7 us against 2 - 3).
constexpr int kSimtK = 32;

void gemm(const Op& a, const Op& b, const float* bias, int act, void* out, ll ldc, bool out_bf16, bool accumulate,
          void* act_grad, const Tensor* like, bool tf32, bool splits) {
  const int M = static_cast<int>(a.rows), N = static_cast<int>(b.rows), K = static_cast<int>(a.k);
  TORCH_CHECK(a.k == b.k, "inner dimensions differ: [", a.rows, ", ", a.k, "] x [", b.rows, ", ", b.k, "]^T");
  TORCH_CHECK(a.bf16 == b.bf16, "gemm: operands of two types");
  TORCH_CHECK(!(out_bf16 && accumulate), "gemm: nothing accumulates onto a bf16 result");
  TORCH_CHECK(a.bf16 || !out_bf16, "gemm: fp32 operands have an fp32 result");
  TORCH_CHECK(act <= FB_ACT_SIGMOID, "gemm: no epilogue evaluates activation ", act);
  if (M == 0 || N == 0) return;
  const bool ok = tma_ok(a) && tma_ok(b);
  const int a_mn = a.s_k == 1 ? 0 : 1, b_mn = b.s_k == 1 ? 0 : 1;
  const ll lda = a_mn ? a.s_k : a.s_row, ldb = b_mn ? b.s_k : b.s_row;
  if (a.bf16 && ok) {
    if (g_max_ctas.load(std::memory_order_relaxed) == 0) {
      if (splits && fb_gemm_bf16_splitk_use(M, N, K)) {
        FB_CALL(fb_gemm_bf16_splitk, a.p, b.p, out, act_grad, bias, M, N, K, lda, ldb, ldc, a_mn, b_mn, out_bf16, act,
                accumulate, 0, status(), cur_stream());
        return;
      }
      if (fb_gemm_bf16_narrow_use(M, N, K)) {
        FB_CALL(fb_gemm_bf16_narrow, a.p, b.p, out, act_grad, bias, M, N, K, lda, ldb, ldc, a_mn, b_mn, out_bf16, act,
                accumulate, 0, status(), cur_stream());
        return;
      }
    }
    int rc = -3;
    if (g_use_2cta.load(std::memory_order_relaxed) && M >= 512 && N >= 128)
      launch("fb_gemm_bf16", [&] {
        rc = fb_gemm_bf16_2cta(a.p, b.p, out, act_grad, bias, M, N, K, lda, ldb, ldc, a_mn, b_mn, out_bf16, act,
                               accumulate, g_max_ctas, status(), cur_stream());
        return rc == -3 ? 0 : rc;  // -3: CTA pairs cannot be scheduled on this device
      });
    if (rc == -3)
      FB_CALL(fb_gemm_bf16, a.p, b.p, out, act_grad, bias, M, N, K, lda, ldb, ldc, a_mn, b_mn, out_bf16, act,
              accumulate, g_max_ctas, status(), cur_stream());
    return;
  }
  TORCH_CHECK(act_grad == nullptr, "activation derivatives need operands that a TMA map describes");
  if (tf32 && ok) {
    int rc = -3;
    if (M >= 512 && N >= 256)
      launch("fb_gemm_tf32", [&] {
        rc = fb_gemm_tf32_2cta(static_cast<const float*>(a.p), static_cast<const float*>(b.p), static_cast<float*>(out),
                               bias, M, N, K, lda, ldb, ldc, a_mn, b_mn, act, accumulate, g_max_ctas, status(), cur_stream());
        return rc == -3 ? 0 : rc;
      });
    if (rc == -3)
      FB_CALL(fb_gemm_tf32, static_cast<const float*>(a.p), static_cast<const float*>(b.p), static_cast<float*>(out),
              bias, M, N, K, lda, ldb, ldc, a_mn, b_mn, act, accumulate, g_max_ctas, status(), cur_stream());
    return;
  }
  if (a.bf16) {  // operands that a TMA map cannot describe
    const bool rows_tma = reinterpret_cast<uintptr_t>(out) % 16 == 0 && ldc * (out_bf16 ? 2 : 4) % 16 == 0;
    if (like != nullptr && (copies_repay(a, b, rows_tma) || (out_bf16 && repack_repays(a, b)))) {
      Tensor ka, kb;
      Op pa = a, pb = b;
      aligned_copies(pa, pb, like->options().dtype(at::kBFloat16).requires_grad(false), ka, kb);
      gemm(pa, pb, bias, act, out, ldc, out_bf16, accumulate, nullptr, like, tf32, splits);
      return;
    }
    FB_CALL(fb_gemm_bf16_any, a.p, b.p, out, bias, M, N, K, a.s_row, a.s_k, b.s_row, b.s_k, ldc, out_bf16, act,
            accumulate, status(), cur_stream());
    return;
  }
  if (K > kSimtK) {
    FB_CALL(fb_gemm_f32_tensor, static_cast<const float*>(a.p), static_cast<const float*>(b.p), static_cast<float*>(out),
            bias, M, N, K, a.s_row, a.s_k, b.s_row, b.s_k, ldc, act, accumulate, 1.f, 1, 1, 0, 0, 0, 0, 0, 0, status(),
            cur_stream());
    return;
  }
  FB_CALL(fb_gemm_f32_simt, static_cast<const float*>(a.p), static_cast<const float*>(b.p), static_cast<float*>(out), bias,
          M, N, K, a.s_row, a.s_k, b.s_k, b.s_row, ldc, act, accumulate, 1, 0, 0, 0, cur_stream());
}

// --------------------------------------------------------------------------------------------------- sinks
Sink::~Sink() {
  if (sink != nullptr && Py_IsInitialized()) {
    py::gil_scoped_acquire gil;
    Py_XDECREF(sink);
    Py_XDECREF(param);
  }
}
std::shared_ptr<Sink> make_sink(py::handle sink, py::handle param) {
  if (sink.is_none()) return nullptr;
  auto s = std::make_shared<Sink>();
  s->sink = sink.inc_ref().ptr();
  s->param = param.inc_ref().ptr();
  return s;
}
void wgrad_to_sink(Sink& s, const Tensor& g2, const Tensor& x2) {
  Tensor buf;
  bool acc = false;
  {
    py::gil_scoped_acquire gil;
    py::handle sink(s.sink), param(s.param);
    if (is_bf16(g2) && is_bf16(x2) && py::hasattr(sink, "try_push") &&
        sink.attr("try_push")(param, g2.t(), x2.t()).cast<bool>())
      return;
    py::tuple r = sink.attr("acquire")(param);
    buf = r[0].cast<Tensor>();
    acc = r[1].cast<bool>();
  }
  gemm(op2d(g2).t(), op2d(x2).t(), nullptr, 0, buf.data_ptr(), buf.stride(0), false, acc, nullptr, &g2,
       g_tf32.load(std::memory_order_relaxed), true);
}
void sink_ready(Sink& s) {
  py::gil_scoped_acquire gil;
  py::handle(s.sink).attr("ready")(py::handle(s.param));
}

}  // namespace fbn

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  using namespace fbn;
  m.def("launch_count", [] { return g_launches.load(); });
  m.def("set_tf32", [](bool f) { g_tf32 = f; });
  m.def("set_use_2cta", [](bool f) { g_use_2cta = f; });
  m.def("set_max_ctas", [](int n) { g_max_ctas = n; });
  m.def("profile_start", [] {
    std::lock_guard<std::mutex> lock(g_prof_mutex);
    for (auto& r : g_records) {
      fb_rt_event_destroy(r.e0);
      fb_rt_event_destroy(r.e1);
    }
    g_records.clear();
    g_profiling = true;
  });
  m.def("profile_stop", [] { g_profiling = false; });
  m.def("profile_records", [] {  // (launcher, milliseconds) of every call since profile_start; synchronizes
    std::vector<std::pair<std::string, float>> out;
    std::lock_guard<std::mutex> lock(g_prof_mutex);
    for (auto& r : g_records) {
      fb_rt_event_synchronize(r.e1);
      out.emplace_back(r.name, fb_rt_event_elapsed_ms(r.e0, r.e1));
    }
    return out;
  });
  m.def("cast", [](const Tensor& t, const Tensor& like) { return cast(t, like.scalar_type()); });
  bind_linear(m);
  bind_elementwise(m);
  bind_layers(m);
  bind_conv(m);
  bind_optim(m);
}
