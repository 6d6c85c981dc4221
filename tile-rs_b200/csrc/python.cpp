// The typed operators for CPython: plain integers (and a float) in, a status out, without building ctypes structures and arguments on
// every call.  A call of a small operator is mostly host time: softmax of 256 x 1000 in a row of calls, see hal.py.
//
// bind(addresses) takes the library's entry points in the order of `Entry`; every other function answers the entry point's status, or
// None where an argument is not a plain int in the range of its field (or float), so that the caller can go through ctypes, which has
// rules of its own for those.  The interpreter lock is released during the call, as ctypes does.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstdint>

#include "../../include/tile_sm100.h"

namespace {

enum Entry { kSoftmax, kRmsNorm, kSiluMul, kGemm, kAttention, kRope, kKvCacheUpdate, kPrefill, kDecode, kEntries };
void* g_entry[kEntries] = {};

// Walks through the arguments; `ok` turns false at the first that does not fit.
struct Args {
  PyObject* const* at;
  Py_ssize_t left;
  bool ok;
  Args(PyObject* const* args, Py_ssize_t n, Py_ssize_t want, Entry e) : at(args), left(n), ok(n == want && g_entry[e] != nullptr) {}
  int64_t i64() {
    if (!ok || left <= 0 || !PyLong_CheckExact(*at)) {
      ok = false;
      return 0;
    }
    int over = 0;
    const long long v = PyLong_AsLongLongAndOverflow(*at, &over);
    ++at, --left;
    if (over) ok = false;
    return v;
  }
  int32_t i32() {
    const int64_t v = i64();
    if (v < INT32_MIN || v > INT32_MAX) ok = false;
    return static_cast<int32_t>(v);
  }
  template <typename T = void>
  T* ptr() {
    if (!ok || left <= 0 || !PyLong_CheckExact(*at)) {
      ok = false;
      return nullptr;
    }
    const unsigned long long v = PyLong_AsUnsignedLongLong(*at);
    ++at, --left;
    if (v == static_cast<unsigned long long>(-1) && PyErr_Occurred()) {
      PyErr_Clear();
      ok = false;
    }
    return reinterpret_cast<T*>(static_cast<uintptr_t>(v));
  }
  float f32() {
    if (!ok || left <= 0 || !PyFloat_CheckExact(*at)) {
      ok = false;
      return 0.f;
    }
    --left;
    return static_cast<float>(PyFloat_AS_DOUBLE(*at++));
  }
};

template <typename Fn, typename... A>
PyObject* call(const Args& args, Entry e, A... a) {
  if (!args.ok) Py_RETURN_NONE;
  int32_t st;
  Py_BEGIN_ALLOW_THREADS
  st = reinterpret_cast<Fn>(g_entry[e])(a...);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(st);
}

PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != kEntries) {
    PyErr_SetString(PyExc_TypeError, "bind: one address per entry point");
    return nullptr;
  }
  for (int i = 0; i < kEntries; ++i) {
    void* p = PyLong_AsVoidPtr(args[i]);
    if (!p && PyErr_Occurred()) return nullptr;
    g_entry[i] = p;
  }
  Py_RETURN_NONE;
}

// (device, dtype, rows, cols, x, y, stream)
PyObject* softmax(PyObject*, PyObject* const* args, Py_ssize_t n) {
  Args a(args, n, 7, kSoftmax);
  auto* dev = a.ptr<tsm100_device_s>();
  tsm100_softmax_desc d = {};
  d.dtype = a.i32(), d.rows = a.i64(), d.cols = a.i64();
  void *x = a.ptr(), *y = a.ptr(), *s = a.ptr();
  return call<decltype(&tsm100_softmax)>(a, kSoftmax, dev, &d, x, y, s);
}
// (device, dtype, rows, cols, eps, x, y, stream)
PyObject* rms_norm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  Args a(args, n, 8, kRmsNorm);
  auto* dev = a.ptr<tsm100_device_s>();
  tsm100_rms_norm_desc d = {};
  d.dtype = a.i32(), d.rows = a.i64(), d.cols = a.i64(), d.eps = a.f32();
  void *x = a.ptr(), *y = a.ptr(), *s = a.ptr();
  return call<decltype(&tsm100_rms_norm)>(a, kRmsNorm, dev, &d, x, y, s);
}
// (device, dtype, rows, cols, gate, up, y, stream)
PyObject* silu_mul(PyObject*, PyObject* const* args, Py_ssize_t n) {
  Args a(args, n, 8, kSiluMul);
  auto* dev = a.ptr<tsm100_device_s>();
  tsm100_silu_mul_desc d = {};
  d.dtype = a.i32(), d.rows = a.i64(), d.cols = a.i64();
  void *gate = a.ptr(), *up = a.ptr(), *y = a.ptr(), *s = a.ptr();
  return call<decltype(&tsm100_silu_mul)>(a, kSiluMul, dev, &d, gate, up, y, s);
}
// (device, dtype, out_dtype, b_transposed, batch, m, n, k, lda, ldb, ldc, a, b, c, stream)
PyObject* gemm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  Args a(args, n, 15, kGemm);
  auto* dev = a.ptr<tsm100_device_s>();
  tsm100_gemm_desc d = {};
  d.dtype = a.i32(), d.out_dtype = a.i32(), d.b_transposed = a.i32(), d.batch = a.i32();
  d.m = a.i64(), d.n = a.i64(), d.k = a.i64(), d.lda = a.i64(), d.ldb = a.i64(), d.ldc = a.i64();
  void *x = a.ptr(), *y = a.ptr(), *c = a.ptr(), *s = a.ptr();
  return call<decltype(&tsm100_gemm)>(a, kGemm, dev, &d, x, y, c, s);
}
// (device, dtype, causal, batch, heads_q, heads_kv, seq, head_dim, q, k, v, o, stream)
PyObject* attention(PyObject*, PyObject* const* args, Py_ssize_t n) {
  Args a(args, n, 13, kAttention);
  auto* dev = a.ptr<tsm100_device_s>();
  tsm100_attention_desc d = {};
  d.dtype = a.i32(), d.causal = a.i32(), d.batch = a.i32(), d.heads_q = a.i32(), d.heads_kv = a.i32(), d.seq = a.i32(), d.head_dim = a.i32();
  void *q = a.ptr(), *k = a.ptr(), *v = a.ptr(), *o = a.ptr(), *s = a.ptr();
  return call<decltype(&tsm100_attention)>(a, kAttention, dev, &d, q, k, v, o, s);
}
// (device, dtype, batch, seq_len, heads, head_dim, start_pos, theta, x, stream)
PyObject* rope(PyObject*, PyObject* const* args, Py_ssize_t n) {
  Args a(args, n, 10, kRope);
  auto* dev = a.ptr<tsm100_device_s>();
  tsm100_rope_desc d = {};
  d.dtype = a.i32(), d.batch = a.i32(), d.seq_len = a.i32(), d.heads = a.i32(), d.head_dim = a.i32(), d.start_pos = a.i32(), d.theta = a.f32();
  void *x = a.ptr(), *s = a.ptr();
  return call<decltype(&tsm100_rope)>(a, kRope, dev, &d, x, s);
}
// (device, dtype, batch, seq_len, heads, head_dim, start_pos, max_seq, src, cache, stream)
PyObject* kv_cache_update(PyObject*, PyObject* const* args, Py_ssize_t n) {
  Args a(args, n, 11, kKvCacheUpdate);
  auto* dev = a.ptr<tsm100_device_s>();
  tsm100_kv_cache_update_desc d = {};
  d.dtype = a.i32(), d.batch = a.i32(), d.seq_len = a.i32(), d.heads = a.i32(), d.head_dim = a.i32(), d.start_pos = a.i32(), d.max_seq = a.i32();
  void *src = a.ptr(), *cache = a.ptr(), *s = a.ptr();
  return call<decltype(&tsm100_kv_cache_update)>(a, kKvCacheUpdate, dev, &d, src, cache, s);
}
// (device, dtype, heads_q, heads_kv, seq_len, start_pos, max_seq, head_dim, q, k_cache, v_cache, o, stream)
PyObject* attention_prefill(PyObject*, PyObject* const* args, Py_ssize_t n) {
  Args a(args, n, 13, kPrefill);
  auto* dev = a.ptr<tsm100_device_s>();
  tsm100_attention_prefill_desc d = {};
  d.dtype = a.i32(), d.heads_q = a.i32(), d.heads_kv = a.i32(), d.seq_len = a.i32(), d.start_pos = a.i32(), d.max_seq = a.i32(), d.head_dim = a.i32();
  void *q = a.ptr(), *k = a.ptr(), *v = a.ptr(), *o = a.ptr(), *s = a.ptr();
  return call<decltype(&tsm100_attention_prefill)>(a, kPrefill, dev, &d, q, k, v, o, s);
}
// (device, dtype, batch, heads_q, heads_kv, seq_len, max_seq, head_dim, q, k_cache, v_cache, o, stream)
PyObject* attention_decode(PyObject*, PyObject* const* args, Py_ssize_t n) {
  Args a(args, n, 13, kDecode);
  auto* dev = a.ptr<tsm100_device_s>();
  tsm100_attention_decode_desc d = {};
  d.dtype = a.i32(), d.batch = a.i32(), d.heads_q = a.i32(), d.heads_kv = a.i32(), d.seq_len = a.i32(), d.max_seq = a.i32(), d.head_dim = a.i32();
  void *q = a.ptr(), *k = a.ptr(), *v = a.ptr(), *o = a.ptr(), *s = a.ptr();
  return call<decltype(&tsm100_attention_decode)>(a, kDecode, dev, &d, q, k, v, o, s);
}

#define TSM_METHOD(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {TSM_METHOD(bind), TSM_METHOD(softmax), TSM_METHOD(rms_norm), TSM_METHOD(silu_mul), TSM_METHOD(gemm), TSM_METHOD(attention),
                           TSM_METHOD(rope), TSM_METHOD(kv_cache_update), TSM_METHOD(attention_prefill), TSM_METHOD(attention_decode),
                           {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_tile_sm100", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__tile_sm100(void) { return PyModule_Create(&g_module); }
