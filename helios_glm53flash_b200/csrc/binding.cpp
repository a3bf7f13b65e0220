// CPython binding of the hk_* entry points that a decode step calls over and over.
//
// A launch costs the host about 2 us; through ctypes the same call cost 10-15 us more (one c_void_p object per tensor, the
// argtypes conversion of 20-30 arguments, a torch Stream object per call), which made every decode call host-bound
// (the KDA layer of one token: 17.2 us per call around a 5.4 us kernel; with this binding 5.5 us).  Here a call is one
// METH_FASTCALL function: tensors are unwrapped to their addresses and the numbers converted straight into the C call.
//
// Conversion rules, by the C type of the parameter:
//   pointer        tensor (or another object with data_ptr()) -> its address, None -> NULL; a tensor that has no address
//                  (sparse, wrapped by a transform) raises the RuntimeError of Tensor.data_ptr()
//   void* stream   (last parameter of a launcher) None -> torch's current stream, torch Stream -> its handle
//   int            int / bool; a tensor gives the dtype tag HK_F16 / HK_BF16 / HK_F32
//   int64_t        int; a [rows][512] tensor gives its row count, 0 if it is not laid out that way
//   size_t         int; a tensor gives its element count (byte workspaces), None gives 0
//   float          number
// The functions return what the C function returns (launchers: the hk_status).  The addresses come from the library that
// the Python layer loaded (bind), so that both sides drive the same build.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <c10/cuda/CUDAStream.h>
#include <c10/util/Exception.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>
#include <exception>
#include <tuple>
#include <type_traits>
#include <utility>

#include "../../include/helios_b200.h"

namespace {

bool bad_arg(const char* what) {
  PyErr_SetString(PyExc_TypeError, what);
  return false;
}

bool number(PyObject* o, long long& v) {
  v = PyLong_AsLongLong(o);
  return !(v == -1 && PyErr_Occurred());
}

template <class T>
bool convert(PyObject* o, T& v) {
  if constexpr (std::is_pointer_v<T>) {
    if (o == Py_None) {
      v = nullptr;
      return true;
    }
    if (THPVariable_Check(o)) {
      const at::Tensor& t = THPVariable_Unpack(o);
      // what the call writes is asked for as such: a lazily cloned tensor gets memory of its own first
      if constexpr (std::is_const_v<std::remove_pointer_t<T>>) v = reinterpret_cast<T>(t.const_data_ptr());
      else v = reinterpret_cast<T>(t.mutable_data_ptr());
      return true;
    }
    PyObject* a = PyObject_CallMethod(o, "data_ptr", nullptr);
    if (!a) return false;
    v = reinterpret_cast<T>(PyLong_AsVoidPtr(a));
    Py_DECREF(a);
    return !PyErr_Occurred();
  } else if constexpr (std::is_floating_point_v<T>) {
    const double d = PyFloat_AsDouble(o);
    if (d == -1.0 && PyErr_Occurred()) return false;
    v = static_cast<T>(d);
    return true;
  } else {
    if (THPVariable_Check(o)) {
      const at::Tensor& t = THPVariable_Unpack(o);
      if constexpr (std::is_same_v<T, int>) {
        switch (t.scalar_type()) {
          case at::kHalf: v = HK_F16; return true;
          case at::kBFloat16: v = HK_BF16; return true;
          case at::kFloat: v = HK_F32; return true;
          default: return bad_arg("tensor dtype: float16, bfloat16 or float32");
        }
      } else if constexpr (std::is_same_v<T, size_t>) {
        v = static_cast<T>(t.numel());
      } else {
        v = t.dim() >= 1 && t.numel() % 512 == 0 ? static_cast<T>(t.numel() / 512) : 0;
      }
      return true;
    }
    if constexpr (std::is_same_v<T, size_t>) {
      if (o == Py_None) {
        v = 0;
        return true;
      }
    }
    long long n;
    if (!number(o, n)) return false;
    if constexpr (std::is_same_v<T, int>) {
      if (n < INT32_MIN || n > INT32_MAX) return bad_arg("integer argument out of range");
    }
    v = static_cast<T>(n);
    return true;
  }
}

bool convert_stream(PyObject* o, void*& v) {
  if (o == Py_None) {
    try {
      v = c10::cuda::getCurrentCUDAStream().stream();
    } catch (const std::exception&) {
      PyErr_SetString(PyExc_RuntimeError, "helios_glm53flash_b200 needs a CUDA device (sm_100a); there is no CPU path");
      return false;
    }
    return true;
  }
  PyObject* h = PyObject_GetAttrString(o, "cuda_stream");
  if (!h) return false;
  v = PyLong_AsVoidPtr(h);
  Py_DECREF(h);
  return !PyErr_Occurred();
}

template <bool STREAM, size_t I, size_t N, class T>
bool convert_at(PyObject* o, T& v) {
  if constexpr (STREAM && I + 1 == N) return convert_stream(o, v);
  else return convert(o, v);
}

template <bool STREAM, class R, class... A, size_t... I>
PyObject* call(R (*fn)(A...), PyObject* const* args, std::index_sequence<I...>) {
  std::tuple<std::remove_const_t<A>...> v;
  try {
    if (!(convert_at<STREAM, I, sizeof...(A)>(args[I], std::get<I>(v)) && ...)) return nullptr;
  } catch (const c10::Error& e) {          // a tensor without an address: sparse, wrapped by vmap, ...
    PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
    return nullptr;
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
  R r;
  if constexpr (STREAM) {
    Py_BEGIN_ALLOW_THREADS;      // a launch may wait for room in the stream's queue
    r = fn(std::get<I>(v)...);
    Py_END_ALLOW_THREADS;
  } else {
    r = fn(std::get<I>(v)...);
  }
  if constexpr (std::is_same_v<R, size_t>) return PyLong_FromSize_t(r);
  else return PyLong_FromLong(r);
}

template <class F>
struct Entry;
template <class R, class... A>
struct Entry<R (*)(A...)> {
  template <bool STREAM>
  static PyObject* run(R (*fn)(A...), const char* name, PyObject* const* args, Py_ssize_t n) {
    if (!fn) {
      PyErr_SetString(PyExc_RuntimeError, "the binding is not bound to the library");
      return nullptr;
    }
    if (n != (Py_ssize_t)sizeof...(A))
      return PyErr_Format(PyExc_TypeError, "%s takes %d arguments, %d given", name, (int)sizeof...(A), (int)n);
    return call<STREAM>(fn, args, std::index_sequence_for<A...>{});
  }
};

// every entry point: X(name, ends in a stream)
#define HK_ENTRIES(X)                                                                                                       \
  X(hk_conv1d_update, true) X(hk_kda_recurrent, true) X(hk_kda_decode_step, true) X(hk_kda_decode_layer, true)               \
  X(hk_kda_dispatch_is_chunked, false) X(hk_kda_chunked_workspace_bytes, false) X(hk_kda_chunked_prefill, true)              \
  X(hk_kda_chunked_prefill_gated, true) X(hk_kda_transpose_cast, true) X(hk_kda_gate, true) X(hk_kda_prepare, true)          \
  X(hk_kda_cast_conv, true) X(hk_gated_rms_norm, true) X(hk_kpool_write, true) X(hk_indexer_score, true)                     \
  X(hk_indexer_score_legacy, true) X(hk_dsa_topk, true) X(hk_dsa_topk_expand, true) X(hk_indexer_select, true)               \
  X(hk_pool_expand, true) X(hk_mla_partial_bytes, false) X(hk_mla_auto_splits, false) X(hk_mla_sparse, true)                 \
  X(hk_mla_sparse_static, true) X(hk_mla_dense, true) X(hk_mla_dense_partial, true) X(hk_mla_dense_partial_ws, true)         \
  X(hk_lse_combine, true) X(hk_q_latent, true) X(hk_o_absorb, true) X(hk_wuv_transpose, true) X(hk_o_absorb_t, true)         \
  X(hk_q_latent_beside, true) X(hk_o_absorb_beside, true) X(hk_kda_decode_layer_beside, true)                                \
  X(hk_mla_cache_append, true) X(hk_layernorm_f16, true) X(hk_mla_decode_prologue, true)

#define X(name, stream)                                                                      \
  decltype(&::name) p_##name = nullptr;                                                      \
  PyObject* py_##name(PyObject*, PyObject* const* args, Py_ssize_t n) {                      \
    return Entry<decltype(&::name)>::run<stream>(p_##name, #name, args, n);                  \
  }
HK_ENTRIES(X)
#undef X

// bind(dict name -> address)
PyObject* py_bind(PyObject*, PyObject* d) {
  if (!PyDict_Check(d)) {
    bad_arg("bind: a dict of addresses");
    return nullptr;
  }
#define X(name, stream)                                                                       \
  {                                                                                           \
    PyObject* a = PyDict_GetItemString(d, #name);                                             \
    if (!a) return PyErr_Format(PyExc_KeyError, "%s", #name);                                 \
    void* p = PyLong_AsVoidPtr(a);                                                            \
    if (PyErr_Occurred()) return nullptr;                                                     \
    p_##name = reinterpret_cast<decltype(p_##name)>(p);                                       \
  }
  HK_ENTRIES(X)
#undef X
  Py_RETURN_NONE;
}

#define X(name, stream) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_##name)), METH_FASTCALL, nullptr},
PyMethodDef methods[] = {HK_ENTRIES(X){"bind", py_bind, METH_O, nullptr}, {nullptr, nullptr, 0, nullptr}};
#undef X

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_binding", "native call path of the hk_* entry points", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__binding(void) { return PyModule_Create(&module); }
