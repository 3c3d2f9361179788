// Python bindings of the native ops and layers: METH_FASTCALL functions whose argument conversions are derived from the
// C++ signatures.
#include <Python.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <dlfcn.h>

#include "native_layers.h"

namespace exb {
namespace {

PyObject* g_library_error = nullptr;   // exact_b200.ExactB200Error

// ---- Python -> C++ ------------------------------------------------------------------------------------
const Tensor& tensor_of(PyObject* o) {
  if (!THPVariable_Check(o)) throw std::runtime_error("expected a tensor, got " + std::string(Py_TYPE(o)->tp_name));
  return THPVariable_Unpack(o);
}
template <class T>
struct Arg;
template <>
struct Arg<Tensor> {
  static const Tensor& get(PyObject* o) { return tensor_of(o); }
};
template <>
struct Arg<OptTensor> {
  static OptTensor get(PyObject* o) { return o == Py_None ? OptTensor() : OptTensor(tensor_of(o)); }
};
template <>
struct Arg<int64_t> {
  static int64_t get(PyObject* o) {
    const int64_t v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw python_error();
    return v;
  }
};
template <>
struct Arg<uint64_t> {
  static uint64_t get(PyObject* o) {
    const uint64_t v = PyLong_AsUnsignedLongLongMask(o);
    if (v == (uint64_t)-1 && PyErr_Occurred()) throw python_error();
    return v;
  }
};
template <>
struct Arg<double> {
  static double get(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw python_error();
    return v;
  }
};
template <>
struct Arg<bool> {
  static bool get(PyObject* o) { return PyObject_IsTrue(o) == 1; }
};
template <class T>
struct Capsule;   // name of a C++ object that travels as a capsule
template <>
struct Capsule<PlanPtr> { static constexpr const char* name = "exact_b200.RowPlan"; };
template <>
struct Capsule<c10::intrusive_ptr<Graph>> { static constexpr const char* name = "exact_b200.Graph"; };
template <class T>
T& capsule_of(PyObject* o) {
  void* p = PyCapsule_GetPointer(o, Capsule<T>::name);
  if (p == nullptr) throw python_error();
  return *static_cast<T*>(p);
}
template <class T>
PyObject* make_capsule(T value) {
  return PyCapsule_New(new T(std::move(value)), Capsule<T>::name,
                       [](PyObject* o) { delete static_cast<T*>(PyCapsule_GetPointer(o, Capsule<T>::name)); });
}
template <>
struct Arg<PlanPtr> {
  static const PlanPtr& get(PyObject* o) { return capsule_of<PlanPtr>(o); }
};
template <>
struct Arg<c10::intrusive_ptr<Graph>> {
  static const c10::intrusive_ptr<Graph>& get(PyObject* o) { return capsule_of<c10::intrusive_ptr<Graph>>(o); }
};

// ---- C++ -> Python ------------------------------------------------------------------------------------
PyObject* to_py(const Tensor& t) {
  if (!t.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(t);
}
PyObject* to_py(int64_t v) { return PyLong_FromLongLong(v); }
PyObject* to_py(bool v) { return PyBool_FromLong(v); }
PyObject* to_py(PyObject* o) { return o; }
PyObject* tuple_of(std::initializer_list<const Tensor*> ts) {
  PyObject* r = PyTuple_New((Py_ssize_t)ts.size());
  Py_ssize_t i = 0;
  for (const Tensor* t : ts) PyTuple_SET_ITEM(r, i++, to_py(*t));
  return r;
}
PyObject* to_py(const Packed& q) { return tuple_of({&q.codes, &q.scale, &q.mn}); }
PyObject* to_py(const std::tuple<Tensor, Tensor>& t) { return tuple_of({&std::get<0>(t), &std::get<1>(t)}); }

PyObject* to_py(const std::tuple<Tensor, Tensor, Tensor>& t) { return tuple_of({&std::get<0>(t), &std::get<1>(t), &std::get<2>(t)}); }

template <class F>
struct Fast;
template <class R, class... A>
struct Fast<R (*)(A...)> {
  template <R (*fn)(A...), size_t... I>
  static PyObject* run(PyObject* const* args, std::index_sequence<I...>) {
    return to_py(fn(Arg<std::decay_t<A>>::get(args[I])...));
  }
  template <R (*fn)(A...)>
  static PyObject* call(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    try {
      if (n != (Py_ssize_t)sizeof...(A))
        throw std::runtime_error("expected " + std::to_string(sizeof...(A)) + " arguments, got " + std::to_string(n));
      return run<fn>(args, std::index_sequence_for<A...>());
    } catch (const LibraryError& e) {
      PyErr_SetString(g_library_error ? g_library_error : PyExc_RuntimeError, e.what());
      return nullptr;
    }
    END_HANDLE_TH_ERRORS
  }
};
#define EXB_METHOD(name, fn) \
  { name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&Fast<decltype(&fn)>::call<&fn>)), METH_FASTCALL, nullptr }

// ---- functions with shapes of their own ------------------------------------------------------------------
int64_t launches() { return acct.launches.load(); }
bool set_timing(bool on) {
  const bool was = acct.timing.exchange(on);
  if (on) {
    std::lock_guard<std::mutex> lock(acct.mu);
    for (TimedCall& c : acct.calls) {
      cudaEventDestroy(c.begin);
      cudaEventDestroy(c.end);
    }
    acct.calls.clear();
  }
  return was;
}
// [(name, ms, bytes, l2_bytes, edge_columns, flops)] of the calls since the last set_timing(True) or take_calls().
// The caller has synchronised.
PyObject* take_calls() {
  std::vector<TimedCall> calls;
  {
    std::lock_guard<std::mutex> lock(acct.mu);
    calls.swap(acct.calls);
  }
  PyObject* list = PyList_New(0);
  for (TimedCall& c : calls) {
    float ms = 0;
    cudaEventElapsedTime(&ms, c.begin, c.end);
    cudaEventDestroy(c.begin);
    cudaEventDestroy(c.end);
    PyObject* t = Py_BuildValue("(sdLLLd)", c.name, (double)ms, (long long)c.bytes, (long long)c.l2_bytes, (long long)c.edge_columns,
                                c.flops);
    PyList_Append(list, t);
    Py_DECREF(t);
  }
  return list;
}
bool set_clock(bool on) {
  acct.host_ns = 0;
  acct.host_calls = 0;
  return acct.clock.exchange(on);
}
int64_t host_ns() { return acct.host_ns.load(); }
int64_t host_calls() { return acct.host_calls.load(); }
// whether kernels with bounded waits ran on the device since the last call
bool take_status_pending(int64_t device) {
  const uint64_t bit = 1ull << (device & 63);
  return (acct.status_pending.fetch_and(~bit) & bit) != 0;
}

int64_t peek_status(int64_t device) {
  c10::cuda::CUDAGuard guard((c10::DeviceIndex)device);
  int word = 0;
  const int rc = lib.exact_status_peek(&word);
  if (rc != 0) library_failure("exact_status_peek", rc);
  return word;
}

PyObject* make_plan(int64_t threshold, int64_t threshold_f16) {
  auto a = std::make_shared<RowPlan>();
  a->threshold = threshold;
  a->threshold_f16 = threshold_f16;
  return make_capsule(PlanPtr(std::move(a)));
}
// t_rowptr, t_col: the transpose, or None for a graph that is only evaluated
PyObject* make_graph(const Tensor& rowptr, const Tensor& col, const OptTensor& value, const PlanPtr& plan, const OptTensor& t_rowptr,
                     const OptTensor& t_col, const OptTensor& t_value, const PlanPtr& t_plan, const OptTensor& inv_degree) {
  auto g = c10::make_intrusive<Graph>();
  g->fw = Csr{rowptr, col, value, plan};
  if (t_rowptr) g->bw = Csr{*t_rowptr, *t_col, t_value, t_plan};
  g->inv_degree = inv_degree;
  return make_capsule(std::move(g));
}
Tensor linear_op(const Tensor& a, const Tensor& w, const OptTensor& bias, const OptTensor& a2, const OptTensor& w2,
                 const OptTensor& out, bool accumulate, int64_t k_chunk) {
  return linear(a, w, bias, a2, w2, out, accumulate, k_chunk);
}
Tensor spmm_op(const Tensor& rowptr, const Tensor& col, const PlanPtr& plan, const OptTensor& value, const Tensor& mat, bool mean) {
  return spmm(rowptr, col, *plan, value, mat, mean);
}
PyObject* rp_quantize_pack_op(const Tensor& x, const Tensor& R, int64_t bits, uint64_t seed, uint64_t offset, int64_t row_offset,
                              bool want_projection) {
  Tensor y;
  const Packed q = rp_quantize_pack(x, R, bits, seed, offset, row_offset, want_projection ? &y : nullptr);
  return want_projection ? tuple_of({&q.codes, &q.scale, &q.mn, &y}) : to_py(q);
}
std::tuple<Tensor, Tensor, Tensor> bn_backward_op(const Tensor& g, const Tensor& codes, const Tensor& scale, const Tensor& mn,
                                                  int64_t bits, const OptTensor& weight, const Tensor& mean, const Tensor& invstd,
                                                  bool train, bool want_input, bool want_weight, bool want_bias) {
  return bn_backward(g, Packed{codes, scale, mn}, bits, weight, mean, invstd, train, want_input, want_weight, want_bias);
}
Tensor grad_weight_op(const Tensor& g, int64_t bits, const Tensor& p0, const Tensor& s0, const Tensor& m0, int64_t k0,
                      const OptTensor& p1, const OptTensor& s1, const OptTensor& m1, int64_t k1) {
  const Packed q0{p0, s0, m0};
  if (!p1) return grad_weight(g, bits, q0, k0, nullptr, 0);
  const Packed q1{*p1, *s1, *m1};
  return grad_weight(g, bits, q0, k0, &q1, k1);
}
Tensor gcn_op(const Tensor& x, const Tensor& w, const OptTensor& b, const c10::intrusive_ptr<Graph>& graph, int64_t bits,
              int64_t kept, uint64_t seed, uint64_t offset, int64_t row_offset, bool fused, bool half) {
  return gcn_node(x, w, b, graph, Saving{bits, kept, seed, offset, row_offset, fused}, half);
}
Tensor sage_op(const Tensor& x, const Tensor& w_l, const OptTensor& b_l, const OptTensor& w_r,
               const c10::intrusive_ptr<Graph>& graph, bool mean, int64_t bits, int64_t kept, uint64_t seed, uint64_t offset,
               int64_t row_offset, bool fused, bool projected_first, bool gradient_first) {
  return sage_node(x, w_l, b_l, w_r, graph, mean, Saving{bits, kept, seed, offset, row_offset, fused}, projected_first,
                   gradient_first);
}

Tensor bn_op(const Tensor& x, const OptTensor& weight, const OptTensor& bias, const OptTensor& running_mean,
             const OptTensor& running_var, double momentum, double eps, int64_t bits, uint64_t seed, uint64_t offset,
             int64_t row_offset) {
  return bn_node(x, weight, bias, running_mean, running_var, momentum, eps, Saving{bits, 0, seed, offset, row_offset, true});
}
Tensor bn_act_op(const Tensor& x, const OptTensor& weight, const OptTensor& bias, const OptTensor& running_mean,
                 const OptTensor& running_var, double momentum, double eps, int64_t bits, uint64_t seed, uint64_t offset,
                 int64_t row_offset, double p, uint64_t drop_offset) {
  return bn_act_node(x, weight, bias, running_mean, running_var, momentum, eps, Saving{bits, 0, seed, offset, row_offset, true}, p,
                     drop_offset);
}
Tensor aggregate_op(const Tensor& x, const OptTensor& value, const OptTensor& row, const OptTensor& perm,
                    const c10::intrusive_ptr<Graph>& graph,
                    int64_t reduce, bool keep_x, int64_t bits, int64_t kept, uint64_t seed, uint64_t offset, int64_t row_offset,
                    bool fused) {
  return aggregate_node(x, value, row, perm, graph, reduce, keep_x, Saving{bits, kept, seed, offset, row_offset, fused});
}
std::tuple<Tensor, Tensor> spmm_minmax_op(const Tensor& rowptr, const Tensor& col, const PlanPtr& plan, const OptTensor& value,
                                          const Tensor& mat, bool is_max) {
  return spmm_minmax(rowptr, col, *plan, value, mat, is_max);
}

// bind(path of libexact_b200.so, ExactB200Error)
PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 2) {
    PyErr_SetString(PyExc_TypeError, "bind(path, error type)");
    return nullptr;
  }
  const char* path = PyUnicode_AsUTF8(args[0]);
  if (path == nullptr) return nullptr;
  void* h = dlopen(path, RTLD_NOW | RTLD_LOCAL);
  if (h == nullptr) {
    PyErr_SetString(PyExc_OSError, dlerror());
    return nullptr;
  }
#define EXB_RESOLVE(name)                                                          \
  lib.name = reinterpret_cast<decltype(lib.name)>(dlsym(h, #name));                \
  if (lib.name == nullptr) {                                                       \
    PyErr_SetString(PyExc_AttributeError, "the library does not export " #name);   \
    return nullptr;                                                                \
  }
  EXB_FUNCTIONS(EXB_RESOLVE)
#undef EXB_RESOLVE
  Py_XDECREF(g_library_error);
  Py_INCREF(args[1]);
  g_library_error = args[1];
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&bind)), METH_FASTCALL, nullptr},
    EXB_METHOD("launches", launches), EXB_METHOD("set_timing", set_timing), EXB_METHOD("take_calls", take_calls),
    EXB_METHOD("set_clock", set_clock), EXB_METHOD("host_ns", host_ns), EXB_METHOD("host_calls", host_calls),
    EXB_METHOD("take_status_pending", take_status_pending), EXB_METHOD("peek_status", peek_status), EXB_METHOD("make_plan", make_plan), EXB_METHOD("make_graph", make_graph),
    EXB_METHOD("quantize_pack", quantize_pack), EXB_METHOD("unpack", unpack), EXB_METHOD("rademacher", rademacher),
    EXB_METHOD("rp_quantize_pack", rp_quantize_pack_op), EXB_METHOD("bn_backward", bn_backward_op), EXB_METHOD("linear", linear_op), EXB_METHOD("grad_weight", grad_weight_op), EXB_METHOD("grad_weight_takes", grad_weight_takes),
    EXB_METHOD("rows_scale_colsum", rows_scale_colsum), EXB_METHOD("spmm", spmm_op), EXB_METHOD("act", act_node),
    EXB_METHOD("batch_norm", bn_op), EXB_METHOD("batch_norm_act", bn_act_op), EXB_METHOD("aggregate", aggregate_op), EXB_METHOD("spmm_minmax", spmm_minmax_op),
    EXB_METHOD("spmm_minmax_backward", spmm_minmax_backward), EXB_METHOD("spmm_value_backward", spmm_value_backward),
    EXB_METHOD("gcn", gcn_op), EXB_METHOD("sage", sage_op), EXB_METHOD("gcn_eval", gcn_eval), EXB_METHOD("sage_eval", sage_eval), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace
}  // namespace exb

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&exb::module); }
