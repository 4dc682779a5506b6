// The operators as plain Python functions: what the package's wrappers call in eager mode.
//
// torch.ops finds the overload, matches the arguments to the schema and boxes them before the dispatcher sees them: 2.4 us of
// the 5.3 us that the smallest cast took in the host (B200 host, one allocation and one launch included; 3.7 us from here), and
// the smallest calls are bound by the host.  Here the arguments are checked by their exact Python types and the dispatcher is
// called with them as they are.  Everything that hangs on the dispatcher (fake tensors, autograd, vmap, tracing, profiling)
// therefore stays; what torch.ops does in front of it, __torch_function__ of subclasses and modes and the messages for
// arguments of the wrong type, is left to torch.ops: any call with an argument that is not exactly a tensor, a dtype, a bool,
// an int or None where the operator takes one, or under a torch-function mode, goes there.
#include <torch/csrc/python_headers.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/dispatch/Dispatcher.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>
#include <optional>
#include <tuple>
#include <utility>

namespace {

using at::ScalarType;
using at::Tensor;
using Tensor2 = std::tuple<Tensor, Tensor>;
using Tensor3 = std::tuple<Tensor, Tensor, Tensor>;
using Tensor4 = std::tuple<Tensor, Tensor, Tensor, Tensor>;

struct ReleaseGil {  // as torch.ops does around the operator
  PyThreadState *state = PyEval_SaveThread();
  ~ReleaseGil() { PyEval_RestoreThread(state); }
};

// ---- arguments: false if the object is not exactly what the operator takes --------------------------------------------
bool take(PyObject *o, Tensor &v) {
  if (!THPVariable_CheckExact(o)) return false;
  v = THPVariable_Unpack(o);
  return true;
}
bool take(PyObject *o, std::optional<Tensor> &v) {
  if (o == Py_None) return true;
  if (!THPVariable_CheckExact(o)) return false;
  v = THPVariable_Unpack(o);
  return true;
}
bool take(PyObject *o, ScalarType &v) {
  if (!THPDtype_Check(o)) return false;
  v = reinterpret_cast<THPDtype *>(o)->scalar_type;
  return true;
}
bool take(PyObject *o, bool &v) {
  if (!PyBool_Check(o)) return false;
  v = o == Py_True;
  return true;
}
bool take(PyObject *o, int64_t &v) {
  if (!PyLong_CheckExact(o)) return false;
  int overflow = 0;
  v = PyLong_AsLongLongAndOverflow(o, &overflow);
  return overflow == 0;
}

// ---- results ----------------------------------------------------------------------------------------------------------
PyObject *give(Tensor &&v) { return THPVariable_Wrap(std::move(v)); }
template <typename... Ts>
PyObject *give(std::tuple<Ts...> &&v) {
  PyObject *t = PyTuple_New(sizeof...(Ts));
  if (!t) return nullptr;
  Py_ssize_t i = 0;
  const bool ok = std::apply(
      [&](auto &...x) {
        return ([&] {
          PyObject *o = THPVariable_Wrap(std::move(x));
          if (o) PyTuple_SET_ITEM(t, i++, o);
          return o != nullptr;
        }() && ...);
      },
      v);
  if (!ok) {
    Py_DECREF(t);
    return nullptr;
  }
  return t;
}

// The operator under its name in torch.ops, for the calls that are not taken here.  Looked up once per operator and kept: a
// program with a default device (torch.set_default_device, a torch-function mode) makes every call this way.
PyObject *torch_ops_operator(const char *name) {
  PyObject *torch = PyImport_ImportModule("torch");
  PyObject *ops = torch ? PyObject_GetAttrString(torch, "ops") : nullptr;
  PyObject *ns = ops ? PyObject_GetAttrString(ops, "DrissTorch") : nullptr;
  PyObject *op = ns ? PyObject_GetAttrString(ns, name) : nullptr;
  Py_XDECREF(ns);
  Py_XDECREF(ops);
  Py_XDECREF(torch);
  return op;
}

template <typename R, typename... Args>
struct Operator {
  using Signature = R(Args...);
  template <typename Handle, size_t... I>
  static PyObject *run(const char *name, PyObject **in_torch_ops, const Handle &op, PyObject *const *args, Py_ssize_t n,
                       std::index_sequence<I...>) {
    std::tuple<std::decay_t<Args>...> v{};
    if (n != static_cast<Py_ssize_t>(sizeof...(Args)) || at::impl::torch_function_mode_enabled() || !(take(args[I], std::get<I>(v)) && ...)) {
      if (!*in_torch_ops) *in_torch_ops = torch_ops_operator(name);
      return *in_torch_ops ? PyObject_Vectorcall(*in_torch_ops, args, static_cast<size_t>(n), nullptr) : nullptr;
    }
    auto call = [&] {
      ReleaseGil no_gil;
      return op.call(std::get<I>(v)...);
    };
    return give(call());
  }
};

#define DTQ_DIRECT(NAME, ...)                                                                                              \
  PyObject *NAME(PyObject *, PyObject *const *args, Py_ssize_t n) {                                                        \
    using Op = Operator<__VA_ARGS__>;                                                                                      \
    static PyObject *in_torch_ops = nullptr;                                                                               \
    try {                                                                                                                  \
      static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("DrissTorch::" #NAME, "").typed<Op::Signature>(); \
      return Op::run(#NAME, &in_torch_ops, op, args, n, Arity<Op::Signature>{});                                           \
    } catch (...) {                                                                                                        \
      torch::translate_exception_to_python(std::current_exception());                                                      \
      return nullptr;                                                                                                      \
    }                                                                                                                      \
  }
template <typename S>
struct ArityOf;
template <typename R, typename... Args>
struct ArityOf<R(Args...)> {
  using type = std::index_sequence_for<Args...>;
};
template <typename S>
using Arity = typename ArityOf<S>::type;

// the signatures of register_ops.cpp
DTQ_DIRECT(saturated_cast, Tensor, const Tensor &, const Tensor &, ScalarType, bool)
DTQ_DIRECT(saturated_cast_transposed, Tensor, const Tensor &, const Tensor &, ScalarType)
DTQ_DIRECT(saturated_cast_dual, Tensor2, const Tensor &, const Tensor &, ScalarType)
DTQ_DIRECT(amax, Tensor, const Tensor &)
DTQ_DIRECT(dynamic_scaled_quant, Tensor, const Tensor &, ScalarType)
DTQ_DIRECT(dynamic_scaled_quant_with_scale, Tensor3, const Tensor &, ScalarType)
DTQ_DIRECT(dynamic_scaled_quant_rowwise, Tensor3, const Tensor &, ScalarType)
DTQ_DIRECT(dynamic_scaled_quant_dual, Tensor4, const Tensor &, ScalarType)
DTQ_DIRECT(cast_with_amax, Tensor2, const Tensor &, const Tensor &, ScalarType)
DTQ_DIRECT(cast_with_amax_dual, Tensor3, const Tensor &, const Tensor &, ScalarType)
DTQ_DIRECT(mx_fp8_quantize, Tensor2, Tensor, int64_t, int64_t, bool, ScalarType)
DTQ_DIRECT(mx_fp8_quantize_with_amax, Tensor3, Tensor)
DTQ_DIRECT(mx_fp8_quantize_dual, Tensor4, Tensor, bool)
DTQ_DIRECT(mx_fp8_quantize_blocked, Tensor2, Tensor)
DTQ_DIRECT(mx_fp4_quantize, Tensor2, Tensor, bool)
DTQ_DIRECT(mx_fp8_bf16, Tensor, Tensor, Tensor, Tensor, Tensor)
DTQ_DIRECT(mx_fp4_bf16, Tensor, Tensor, Tensor, Tensor, Tensor)
DTQ_DIRECT(sweep_mm, Tensor, Tensor, Tensor, Tensor, Tensor, std::optional<Tensor>, ScalarType, bool, int64_t, int64_t, int64_t, bool,
           int64_t)
#undef DTQ_DIRECT

#define DTQ_METHOD(NAME) {#NAME, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(NAME)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    DTQ_METHOD(saturated_cast), DTQ_METHOD(saturated_cast_transposed), DTQ_METHOD(saturated_cast_dual), DTQ_METHOD(amax),
    DTQ_METHOD(dynamic_scaled_quant), DTQ_METHOD(dynamic_scaled_quant_with_scale), DTQ_METHOD(dynamic_scaled_quant_rowwise),
    DTQ_METHOD(dynamic_scaled_quant_dual), DTQ_METHOD(cast_with_amax), DTQ_METHOD(cast_with_amax_dual), DTQ_METHOD(mx_fp8_quantize),
    DTQ_METHOD(mx_fp8_quantize_with_amax), DTQ_METHOD(mx_fp8_quantize_dual), DTQ_METHOD(mx_fp8_quantize_blocked),
    DTQ_METHOD(mx_fp4_quantize), DTQ_METHOD(mx_fp8_bf16), DTQ_METHOD(mx_fp4_bf16), DTQ_METHOD(sweep_mm), {nullptr, nullptr, 0, nullptr}};
#undef DTQ_METHOD

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_direct", "torch.ops.DrissTorch without the schema match of torch.ops.", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__direct() { return PyModule_Create(&module); }
