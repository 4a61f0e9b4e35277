// Optimizer steps over lists of parameters and the bf16 weight copies that the step keeps current.
#include "native.h"

#include <torch/csrc/autograd/python_variable.h>

namespace fbn {
namespace {

PyObject* s_dict() {
  static PyObject* s = PyUnicode_InternFromString("__dict__");
  return s;
}
PyObject* s_shadow() {
  static PyObject* s = PyUnicode_InternFromString("_fb_shadow");
  return s;
}
PyObject* s_key() {
  static PyObject* s = PyUnicode_InternFromString("_fb_shadow_key");
  return s;
}

const Tensor& unpack(PyObject* o) {
  TORCH_CHECK_TYPE(THPVariable_Check(o), "expected a tensor");
  return THPVariable_Unpack(o);
}

bool key_matches(PyObject* key, const Tensor& p) {
  if (key == nullptr || !PyTuple_Check(key) || PyTuple_GET_SIZE(key) != 2) return false;
  return PyLong_AsLongLong(PyTuple_GET_ITEM(key, 0)) == static_cast<ll>(p._version()) &&
         PyLong_AsUnsignedLongLong(PyTuple_GET_ITEM(key, 1)) == reinterpret_cast<uintptr_t>(p.data_ptr());
}

// The parameter's bf16 copy if it is current, else nullptr: the owning layer casts again on its next forward pass.
void* current_shadow(PyObject* param, const Tensor& p) {
  py::object d = py::reinterpret_steal<py::object>(PyObject_GetAttr(param, s_dict()));
  if (!d) throw py::error_already_set();
  PyObject* sh = PyDict_GetItem(d.ptr(), s_shadow());
  if (sh == nullptr || sh == Py_None) return nullptr;
  const Tensor& t = unpack(sh);
  if (t.sizes() != p.sizes() || !key_matches(PyDict_GetItem(d.ptr(), s_key()), p)) return nullptr;
  return t.data_ptr();
}

// An up-to-date bf16 copy of an fp32 parameter, kept on the parameter.  A change of the parameter outside the fused
// optimizer kernels (in-place op, swapped storage) shows in its version or address and costs one cast.
py::object low_weight(py::handle param) {
  const Tensor& p = unpack(param.ptr());
  if (!p.is_cuda() || !is_f32(p)) return py::none();
  py::object d = py::reinterpret_steal<py::object>(PyObject_GetAttr(param.ptr(), s_dict()));
  if (!d) throw py::error_already_set();
  PyObject* sh = PyDict_GetItem(d.ptr(), s_shadow());
  if (sh != nullptr && sh != Py_None) {
    const Tensor& t = unpack(sh);
    if (t.sizes() == p.sizes() && t.device() == p.device()) {
      if (key_matches(PyDict_GetItem(d.ptr(), s_key()), p)) return py::reinterpret_borrow<py::object>(sh);
    } else {
      sh = nullptr;
    }
  }
  NoAutograd below;
  Tensor t = sh != nullptr && sh != Py_None ? unpack(sh) : at::empty_like(p, p.options().dtype(at::kBFloat16));
  Tensor src = contig(p);
  FB_CALL(fb_cast, src.data_ptr(), t.data_ptr(), p.numel(), FB_DT_F32, FB_DT_BF16, cur_stream());
  py::object out = sh != nullptr && sh != Py_None ? py::reinterpret_borrow<py::object>(sh) : py::cast(t);
  PyDict_SetItem(d.ptr(), s_shadow(), out.ptr());
  py::tuple key = py::make_tuple(static_cast<ll>(p._version()), reinterpret_cast<uintptr_t>(p.data_ptr()));
  PyDict_SetItem(d.ptr(), s_key(), key.ptr());
  return out;
}

struct Table {
  std::vector<float*> p, a, b;
  std::vector<const float*> g;
  std::vector<void*> sh;
  std::vector<ll> n;
  std::vector<Tensor> keep;
  py::list rest;  // indices that take the tensor path: CPU, other types, not contiguous
};

Tensor state_of(py::list& l, size_t i, const Tensor& p) {
  if (l[i].is_none()) l[i] = py::cast(at::zeros_like(p));
  return unpack(l[i].ptr());
}

// `first` / `second`: lists of optimizer state, filled on first use; either may be None.
Table collect(py::list params, py::object first, py::object second) {
  NoAutograd below;
  Table t;
  const size_t n = params.size();
  t.p.reserve(n);
  t.g.reserve(n);
  t.n.reserve(n);
  for (size_t i = 0; i < n; ++i) {
    PyObject* obj = PyList_GET_ITEM(params.ptr(), static_cast<Py_ssize_t>(i));
    const Tensor& p = unpack(obj);
    const Tensor& g = p.grad();
    if (!g.defined()) continue;
    if (!(p.is_cuda() && is_f32(p) && is_f32(g) && p.is_contiguous() && g.is_contiguous())) {
      t.rest.append(i);
      continue;
    }
    t.p.push_back(p.data_ptr<float>());
    t.g.push_back(g.data_ptr<float>());
    t.n.push_back(p.numel());
    t.sh.push_back(current_shadow(obj, p));
    for (int k = 0; k < 2; ++k) {
      py::object& o = k == 0 ? first : second;
      float* q = nullptr;
      if (!o.is_none()) {
        py::list l = py::reinterpret_borrow<py::list>(o);
        q = state_of(l, i, p).data_ptr<float>();
      }
      (k == 0 ? t.a : t.b).push_back(q);
    }
  }
  return t;
}

py::list adam_step(py::list params, py::object m, py::object v, float lr, float beta1, float beta2, float eps, float wd,
                   float bc1, float bc2, const c10::optional<Tensor>& dyn) {
  Table t = collect(params, m, v);
  const int n = static_cast<int>(t.p.size());
  if (n == 0) return t.rest;
  const fb_adam_hparams h{lr, beta1, beta2, eps, wd, bc1, bc2, 1.f};
  if (dyn.has_value()) {
    float* d = dyn->data_ptr<float>();
    FB_CALL(fb_optim_advance, d, beta1, beta2, cur_stream());
    FB_CALL(fb_adam_multi_dyn, t.p.data(), t.g.data(), t.a.data(), t.b.data(), t.sh.data(), t.n.data(), n, h, d, cur_stream());
  } else {
    FB_CALL(fb_adam_multi, t.p.data(), t.g.data(), t.a.data(), t.b.data(), t.sh.data(), t.n.data(), n, h, cur_stream());
  }
  return t.rest;
}

py::list sgd_step(py::list params, py::object velocity, float lr, float momentum, float wd, bool nesterov, bool first,
                  const c10::optional<Tensor>& dyn) {
  Table t = collect(params, velocity, py::none());
  const int n = static_cast<int>(t.p.size());
  if (n == 0) return t.rest;
  const fb_sgd_hparams h{lr, momentum, wd, 1.f, nesterov ? 1 : 0, first ? 1 : 0};
  if (dyn.has_value())
    FB_CALL(fb_sgd_multi_dyn, t.p.data(), t.g.data(), t.a.data(), t.sh.data(), t.n.data(), n, h, dyn->data_ptr<float>(),
            cur_stream());
  else
    FB_CALL(fb_sgd_multi, t.p.data(), t.g.data(), t.a.data(), t.sh.data(), t.n.data(), n, h, cur_stream());
  return t.rest;
}

void clear_grads(py::list params) {
  for (size_t i = 0; i < params.size(); ++i) {
    const Tensor& p = unpack(PyList_GET_ITEM(params.ptr(), static_cast<Py_ssize_t>(i)));
    p.mutable_grad().reset();
  }
}

}  // namespace

void bind_optim(py::module_& m) {
  m.def("low_weight", &low_weight);
  m.def("adam_step", &adam_step);
  m.def("sgd_step", &sgd_step);
  m.def("clear_grads", &clear_grads);
}

}  // namespace fbn
