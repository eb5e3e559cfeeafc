// CPython entry of the operators' launches.
//
// A decode step is a dozen launches of 2 to 10 us of device time each, and the C side of one (checks,
// tensor map look-up, cudaLaunchKernelEx) takes under 3 us.  Through ctypes a call cost 8.7 us: three
// attribute look-ups per plane, a Stream object for the current stream and libffi's marshalling took
// twice the launch itself.  Here a call reads its tensors directly: 3.15 us a launch of the norm of one
// token, 10.5 us (17.8) a norm and the 8192-row projection behind it.
//
// Only the plain forms are read here: exact torch.Tensor / Parameter planes that are contiguous and on a
// GPU, addresses and sizes as int, divisors as float, the current stream or an address.  Any other
// argument, a wrong argument count and a closed context go to the ctypes call (`general`), which accepts or
// refuses them as it always did.  Nothing is kept from one call to the next.
#define PY_SSIZE_T_CLEAN
#include <torch/csrc/autograd/python_variable.h>

#include <c10/cuda/CUDAStream.h>

#include <array>
#include <tuple>
#include <utility>

#include "../../include/tuisko_sm100.h"

namespace {

PyObject* g_general = nullptr;  // general(name, context, stream, *arguments)
PyObject* g_handle = nullptr;   // interned attribute names
PyObject* g_value = nullptr;
PyObject* g_check = nullptr;

bool plain(PyObject* o, int* out) {
  if (!PyLong_CheckExact(o)) return false;
  *out = static_cast<int>(PyLong_AsUnsignedLongMask(o));  // the mask ctypes applies
  return true;
}

bool plain(PyObject* o, float* out) {
  if (!PyFloat_CheckExact(o)) return false;
  *out = static_cast<float>(PyFloat_AS_DOUBLE(o));
  return true;
}

template <class T>
bool plain(PyObject* o, T** out) {
  if (o == Py_None) {
    *out = nullptr;
    return true;
  }
  if (PyLong_CheckExact(o)) {
    *out = reinterpret_cast<T*>(PyLong_AsUnsignedLongMask(o));
    return true;
  }
  if (!THPVariable_CheckExact(o)) return false;
  try {
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.is_cuda() || !t.is_contiguous()) return false;
    *out = static_cast<T*>(const_cast<void*>(static_cast<const void*>(t.data_ptr())));
    return true;
  } catch (...) {  // a wrapper without storage: the general call reports it
    return false;
  }
}

bool plain_stream(PyObject* o, tk100_stream* out) {
  if (o == Py_None) {
    try {
      *out = static_cast<tk100_stream>(c10::cuda::getCurrentCUDAStream().stream());
      return true;
    } catch (...) {
      return false;
    }
  }
  if (!PyLong_CheckExact(o)) return false;
  *out = reinterpret_cast<tk100_stream>(PyLong_AsUnsignedLongMask(o));
  return true;
}

// The context's handle (a ctypes c_void_p, None once closed).
bool plain_context(PyObject* o, tk100_ctx** out) {
  *out = nullptr;
  PyObject* handle = PyObject_GetAttr(o, g_handle);
  PyObject* value = handle ? PyObject_GetAttr(handle, g_value) : nullptr;
  if (value && PyLong_CheckExact(value)) *out = reinterpret_cast<tk100_ctx*>(PyLong_AsUnsignedLongMask(value));
  Py_XDECREF(value);
  Py_XDECREF(handle);
  if (PyErr_Occurred()) PyErr_Clear();
  return *out != nullptr;
}

PyObject* general(const char* name, PyObject* const* args, Py_ssize_t n) {
  PyObject* all = PyTuple_New(n + 1);
  if (!all) return nullptr;
  PyObject* text = PyUnicode_FromString(name);
  if (!text) {
    Py_DECREF(all);
    return nullptr;
  }
  PyTuple_SET_ITEM(all, 0, text);
  for (Py_ssize_t i = 0; i < n; ++i) {
    Py_INCREF(args[i]);
    PyTuple_SET_ITEM(all, i + 1, args[i]);
  }
  PyObject* r = PyObject_CallObject(g_general, all);
  Py_DECREF(all);
  return r;
}

template <class... A, size_t... I>
PyObject* invoke(const char* name, tk100_status (*fn)(tk100_ctx*, tk100_stream, A...), PyObject* const* args,
                 Py_ssize_t n, std::index_sequence<I...>) {
  tk100_ctx* context = nullptr;
  tk100_stream stream = nullptr;
  std::tuple<A...> values{};
  if (n != static_cast<Py_ssize_t>(sizeof...(A)) + 2 || !(plain(args[I + 2], &std::get<I>(values)) && ...) ||
      !plain_context(args[0], &context) || !plain_stream(args[1], &stream)) {
    return general(name, args, n);
  }
  tk100_status status;
  Py_BEGIN_ALLOW_THREADS;  // as a ctypes call: other threads run while a full launch queue drains
  status = fn(context, stream, std::get<I>(values)...);
  Py_END_ALLOW_THREADS;
  if (status == TK100_OK) Py_RETURN_NONE;
  PyObject* code = PyLong_FromLong(static_cast<long>(status));
  if (!code) return nullptr;
  PyObject* r = PyObject_CallMethodObjArgs(args[0], g_check, code, nullptr);  // raises
  Py_DECREF(code);
  return r;
}

template <class... A>
PyObject* invoke(const char* name, tk100_status (*fn)(tk100_ctx*, tk100_stream, A...), PyObject* const* args,
                 Py_ssize_t n) {
  return invoke(name, fn, args, n, std::index_sequence_for<A...>());
}

#define TK100_LAUNCHES(X)                    \
  X(tk100_rms_norm)                          \
  X(tk100_residual_rms_norm)                 \
  X(tk100_residual_rms_norm_quantize)        \
  X(tk100_residual_rms_norm_quantize_nvfp4)  \
  X(tk100_quantize_activation_e4m3)          \
  X(tk100_fp8_qkv)                           \
  X(tk100_fp8_gdn_input)                     \
  X(tk100_fp8_projection)                    \
  X(tk100_fp8_swiglu)                        \
  X(tk100_fp8_down)                          \
  X(tk100_fp8_gdn_output)                    \
  X(tk100_gdn_prepare)                       \
  X(tk100_gdn_recurrence)                    \
  X(tk100_fp8_lm_head)                       \
  X(tk100_nvfp4_quantize_activation)         \
  X(tk100_nvfp4_gate_up_swiglu)              \
  X(tk100_nvfp4_gate_up_swiglu_quantize)     \
  X(tk100_nvfp4_down)                        \
  X(tk100_nvfp4_down_partial)

#define TK100_WRAPPER(name)                                                              \
  decltype(&::name) g_##name = nullptr;                                                  \
  PyObject* py_##name(PyObject*, PyObject* const* args, Py_ssize_t n) {                  \
    return g_##name ? invoke(#name, g_##name, args, n) : general(#name, args, n);        \
  }
TK100_LAUNCHES(TK100_WRAPPER)

// bind(address_of, general): address_of(name) -> address of the loaded library's function.
PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 2) {
    PyErr_SetString(PyExc_TypeError, "bind(address_of, general)");
    return nullptr;
  }
  Py_INCREF(args[1]);
  Py_XSETREF(g_general, args[1]);
#define TK100_BIND(name)                                                                  \
  {                                                                                       \
    PyObject* address = PyObject_CallFunction(args[0], "s", #name);                       \
    if (!address) return nullptr;                                                         \
    g_##name = reinterpret_cast<decltype(g_##name)>(PyLong_AsVoidPtr(address));           \
    Py_DECREF(address);                                                                   \
    if (PyErr_Occurred()) return nullptr;                                                 \
  }
  TK100_LAUNCHES(TK100_BIND)
  Py_RETURN_NONE;
}

#define TK100_METHOD(name) \
  {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&py_##name)), METH_FASTCALL, nullptr},
PyMethodDef g_methods[] = {
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&bind)), METH_FASTCALL, nullptr},
    TK100_LAUNCHES(TK100_METHOD){nullptr, nullptr, 0, nullptr}};

PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) {
  g_handle = PyUnicode_InternFromString("handle");
  g_value = PyUnicode_InternFromString("value");
  g_check = PyUnicode_InternFromString("check");
  if (!g_handle || !g_value || !g_check) return nullptr;
  return PyModule_Create(&g_module);
}
