// Call path of the small operators without the Python work around a launch: argument checks, the result's
// allocation, the current stream and the C entry point in one extension call.
//
// A decode-sized GEMM (16 x 8192 x 1024) takes 5.2 us with calls in a row; through Python attribute checks,
// `new_empty` and ctypes its call took 8.9 us on the host, of which the entry point (tensor maps and launch) is 4.2.
// A row quantisation takes 5.5 us on the host instead of 10.2.  Every function here
// answers None for whatever it does not recognise - another type, layout or device, a tensor subclass, an
// active dispatch or function mode, a launch that failed - and its caller in ops/ goes on with the general
// path, which knows the errors.  The GIL is released around allocations and launches, which may block.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>

namespace {

using GemmFn = int (*)(const void*, const void*, void*, int, int, int, float, int, int, void*, void*);
using ScaledGemmFn = int (*)(const void*, const void*, const void*, const void*, void*, int, int, int, float,
                             int, int, void*, void*);
using MxGemmFn = int (*)(const void*, const void*, const void*, const void*, void*, int, int, int, float, int,
                         void*, void*);
using QuantFn = int (*)(const void*, void*, void*, long long, int, int, void*);
using QuantPow2Fn = int (*)(const void*, void*, void*, void*, int, long long, int, int, void*);
using AttnFn = int (*)(const void*, const void*, const void*, void*, void*, int, int, int, int, int, int, int,
                       int, float, void*, void*);
using SplitBytesFn = long long (*)(int, int, int, int, int, int, int, int);
using SplitFn = int (*)(const void*, const void*, const void*, void*, void*, int, int, int, int, int, int, int,
                        int, float, void*, long long, void*, void*);

GemmFn g_gemm_bf16, g_gemm_fp8;
ScaledGemmFn g_gemm_bs;
MxGemmFn g_gemm_mx;
QuantFn g_quant;
QuantPow2Fn g_quant_pow2;
AttnFn g_attn;
SplitBytesFn g_split_bytes;
SplitFn g_split;

struct NoGil {
  PyThreadState* s = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(s); }
};

// A plain CUDA tensor that nothing wraps or intercepts, contiguous and 16-byte aligned.
const at::Tensor* plain(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  const auto* impl = t.unsafeGetTensorImpl();
  const auto ks = impl->key_set();
  if (!t.is_cuda() || t.layout() != at::kStrided || ks.has(c10::DispatchKey::Python) ||
      ks.has(c10::DispatchKey::FuncTorchBatched) || ks.has(c10::DispatchKey::FuncTorchGradWrapper) ||
      ks.has(c10::DispatchKey::Functionalize) || ks.has(c10::DispatchKey::Negative) ||
      ks.has(c10::DispatchKey::Conjugate) || ks.has(c10::DispatchKey::ZeroTensor))
    return nullptr;
  if (!t.is_contiguous() || !t.has_storage() || (reinterpret_cast<uintptr_t>(t.const_data_ptr()) & 15u) != 0)
    return nullptr;
  return &t;
}
bool modes_off() {
  return !c10::impl::TorchDispatchModeTLS::any_modes_set() && !at::impl::torch_function_mode_enabled();
}
bool fits(int64_t v) { return v > 0 && v <= 0x7fffffff; }
bool as_int(PyObject* o, int* v) {
  if (!PyLong_CheckExact(o)) return false;
  int over = 0;
  const long long x = PyLong_AsLongLongAndOverflow(o, &over);
  if (over != 0 || x < -0x7fffffffll || x > 0x7fffffffll) return false;
  *v = static_cast<int>(x);
  return true;
}
bool as_ptr(PyObject* o, void** v) {
  if (!PyLong_CheckExact(o)) return false;
  int over = 0;
  const long long x = PyLong_AsLongLongAndOverflow(o, &over);
  if (over != 0 || x < 0) return false;
  *v = reinterpret_cast<void*>(x);
  return true;
}
bool as_float(PyObject* o, float* v) {
  if (!PyFloat_CheckExact(o)) return false;
  *v = static_cast<float>(PyFloat_AS_DOUBLE(o));
  return true;
}
at::Tensor empty(const at::Tensor& like, at::IntArrayRef size, at::ScalarType dt) {
  return at::empty(size, at::TensorOptions().dtype(dt).device(like.device()));
}
// The result of a product: `o` (None: a new one), bf16 [m, n].
bool result(PyObject* o, const at::Tensor& like, int64_t m, int64_t n, at::Tensor* out) {
  if (o == Py_None) {
    NoGil g;
    *out = empty(like, {m, n}, at::kBFloat16);
    return true;
  }
  const at::Tensor* t = plain(o);
  if (t == nullptr || t->dim() != 2 || t->scalar_type() != at::kBFloat16 || t->size(0) != m || t->size(1) != n)
    return false;
  *out = *t;
  return true;
}
void* current_stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
PyObject* give(PyObject* passed, const at::Tensor& out) {
  if (passed == Py_None) return THPVariable_Wrap(out);
  Py_INCREF(passed);
  return passed;
}

#define CB_TRY try {
#define CB_END                  \
  }                             \
  catch (const std::exception&) { \
  }                             \
  Py_RETURN_NONE;

// gemm(a, b, out, alpha, bn, max_ctas, status_ptr)
PyObject* fast_gemm(PyObject*, PyObject* const* v, Py_ssize_t n) {
  CB_TRY
  int bn, max_ctas;
  float alpha;
  void* status;
  if (n != 7 || !modes_off() || !as_float(v[3], &alpha) || !as_int(v[4], &bn) || !as_int(v[5], &max_ctas) ||
      !as_ptr(v[6], &status))
    Py_RETURN_NONE;
  const at::Tensor *a = plain(v[0]), *b = plain(v[1]);
  if (a == nullptr || b == nullptr || a->dim() != 2 || b->dim() != 2) Py_RETURN_NONE;
  const int64_t M = a->size(0), K = a->size(1), N = b->size(0);
  const at::ScalarType dt = a->scalar_type();
  if (b->size(1) != K || b->scalar_type() != dt || !fits(M) || !fits(N) || !fits(K)) Py_RETURN_NONE;
  GemmFn fn = dt == at::kBFloat16 ? g_gemm_bf16 : dt == at::kFloat8_e4m3fn ? g_gemm_fp8 : nullptr;
  at::Tensor out;
  if (fn == nullptr || !result(v[2], *a, M, N, &out)) Py_RETURN_NONE;
  int rc;
  {
    NoGil g;
    rc = fn(a->const_data_ptr(), b->const_data_ptr(), out.mutable_data_ptr(), static_cast<int>(M),
            static_cast<int>(N), static_cast<int>(K), alpha, bn, max_ctas, status, current_stream());
  }
  if (rc == 0) return give(v[2], out);
  CB_END
}

// Shapes of a block-scaled product: e4m3 a [M, K], b [N, K], K a multiple of 128.
bool scaled_shapes(const at::Tensor* a, const at::Tensor* b, int64_t* M, int64_t* N, int64_t* K) {
  if (a == nullptr || b == nullptr || a->dim() != 2 || b->dim() != 2 || a->scalar_type() != at::kFloat8_e4m3fn ||
      b->scalar_type() != at::kFloat8_e4m3fn)
    return false;
  *M = a->size(0);
  *K = a->size(1);
  *N = b->size(0);
  return b->size(1) == *K && *K % 128 == 0 && fits(*M) && fits(*N) && fits(*K);
}
bool is_2d(const at::Tensor* t, at::ScalarType dt, int64_t rows, int64_t cols) {
  return t != nullptr && t->dim() == 2 && t->scalar_type() == dt && t->size(0) == rows && t->size(1) == cols;
}

// gemm_fp8_mx(a_q, a_sf, b_q, b_sf, out, alpha, pair, status_ptr)
PyObject* fast_gemm_mx(PyObject*, PyObject* const* v, Py_ssize_t n) {
  CB_TRY
  float alpha;
  void* status;
  int64_t M, N, K;
  if (n != 8 || !modes_off() || !as_float(v[5], &alpha) || !PyBool_Check(v[6]) || !as_ptr(v[7], &status))
    Py_RETURN_NONE;
  const at::Tensor *a = plain(v[0]), *sa = plain(v[1]), *b = plain(v[2]), *sb = plain(v[3]);
  if (!scaled_shapes(a, b, &M, &N, &K)) Py_RETURN_NONE;
  const int64_t kg = (K / 128 + 3) / 4;
  at::Tensor out;
  if (!is_2d(sa, at::kInt, kg, M) || !is_2d(sb, at::kInt, kg, N) || !result(v[4], *a, M, N, &out))
    Py_RETURN_NONE;
  int rc;
  {
    NoGil g;
    rc = g_gemm_mx(a->const_data_ptr(), sa->const_data_ptr(), b->const_data_ptr(), sb->const_data_ptr(),
                   out.mutable_data_ptr(), static_cast<int>(M), static_cast<int>(N), static_cast<int>(K), alpha,
                   v[6] == Py_True ? 0 : -1, status, current_stream());
  }
  if (rc == 0) return give(v[4], out);
  CB_END
}

// gemm_fp8_blockscaled(a_q, a_s, b_q, b_s, out, alpha, max_ctas, status_ptr)
PyObject* fast_gemm_bs(PyObject*, PyObject* const* v, Py_ssize_t n) {
  CB_TRY
  float alpha;
  void* status;
  int max_ctas;
  int64_t M, N, K;
  if (n != 8 || !modes_off() || !as_float(v[5], &alpha) || !as_int(v[6], &max_ctas) || !as_ptr(v[7], &status))
    Py_RETURN_NONE;
  const at::Tensor *a = plain(v[0]), *sa = plain(v[1]), *b = plain(v[2]), *sb = plain(v[3]);
  if (!scaled_shapes(a, b, &M, &N, &K)) Py_RETURN_NONE;
  at::Tensor out;
  if (!is_2d(sa, at::kFloat, M, K / 128) || !is_2d(sb, at::kFloat, (N + 127) / 128, K / 128) ||
      !result(v[4], *a, M, N, &out))
    Py_RETURN_NONE;
  int rc;
  {
    NoGil g;
    rc = g_gemm_bs(a->const_data_ptr(), sa->const_data_ptr(), b->const_data_ptr(), sb->const_data_ptr(),
                   out.mutable_data_ptr(), static_cast<int>(M), static_cast<int>(N), static_cast<int>(K), alpha, 0,
                   max_ctas, status, current_stream());
  }
  if (rc == 0) return give(v[4], out);
  CB_END
}

// quantize_rows(x, pow2): one scale per row and 128 columns.  (q, scales) or (q, scales, sf).
PyObject* fast_quantize_rows(PyObject*, PyObject* const* v, Py_ssize_t n) {
  CB_TRY
  if (n != 2 || !modes_off() || !PyBool_Check(v[1])) Py_RETURN_NONE;
  const at::Tensor* x = plain(v[0]);
  if (x == nullptr || x->dim() != 2 || x->scalar_type() != at::kBFloat16) Py_RETURN_NONE;
  const int64_t rows = x->size(0), K = x->size(1);
  if (!fits(rows) || !fits(K) || K % 128 != 0) Py_RETURN_NONE;
  const bool pow2 = v[1] == Py_True;
  at::Tensor q, s, sf;
  int rc;
  {
    NoGil g;
    q = empty(*x, {rows, K}, at::kFloat8_e4m3fn);
    s = empty(*x, {rows, K / 128}, at::kFloat);
    if (pow2) {
      sf = empty(*x, {(K / 128 + 3) / 4, rows}, at::kInt);
      rc = g_quant_pow2(x->const_data_ptr(), q.mutable_data_ptr(), s.mutable_data_ptr(), sf.mutable_data_ptr(),
                        static_cast<int>(rows), rows, static_cast<int>(K), 1, current_stream());
    } else {
      rc = g_quant(x->const_data_ptr(), q.mutable_data_ptr(), s.mutable_data_ptr(), rows, static_cast<int>(K), 1,
                   current_stream());
    }
  }
  if (rc == 0) {
    PyObject* t = PyTuple_New(pow2 ? 3 : 2);
    if (t == nullptr) return nullptr;
    PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(q));
    PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(s));
    if (pow2) PyTuple_SET_ITEM(t, 2, THPVariable_Wrap(sf));
    return t;
  }
  CB_END
}

// attention(q, k, v, causal, q_offset, kv_offset, scale | None, status_ptr): new (o, lse).
PyObject* fast_attention(PyObject*, PyObject* const* v, Py_ssize_t n) {
  CB_TRY
  int q_off, kv_off;
  float scale;
  void* status;
  if (n != 8 || !modes_off() || !PyBool_Check(v[3]) || !as_int(v[4], &q_off) || !as_int(v[5], &kv_off) ||
      !as_ptr(v[7], &status))
    Py_RETURN_NONE;
  const at::Tensor *q = plain(v[0]), *k = plain(v[1]), *w = plain(v[2]);
  for (const at::Tensor* t : {q, k, w})
    if (t == nullptr || t->dim() != 4 || t->scalar_type() != at::kBFloat16 || t->size(3) != 128) Py_RETURN_NONE;
  if (v[6] == Py_None) scale = static_cast<float>(1.0 / std::sqrt(128.0));
  else if (!as_float(v[6], &scale)) Py_RETURN_NONE;
  if (w->sizes() != k->sizes() || k->size(0) != q->size(0)) Py_RETURN_NONE;
  const int64_t B = q->size(0), Sq = q->size(1), Hq = q->size(2), Skv = k->size(1), Hkv = k->size(2);
  if (!fits(B) || !fits(Sq) || !fits(Hq) || !fits(Skv) || !fits(Hkv)) Py_RETURN_NONE;
  const int b = static_cast<int>(B), sq = static_cast<int>(Sq), hq = static_cast<int>(Hq),
            skv = static_cast<int>(Skv), hkv = static_cast<int>(Hkv), causal = v[3] == Py_True ? 1 : 0;
  at::Tensor o, lse;
  int rc;
  {
    NoGil g;
    o = empty(*q, q->sizes(), at::kBFloat16);
    lse = empty(*q, {B, Hq, Sq}, at::kFloat);
    const long long ws = g_split_bytes(b, sq, skv, hq, hkv, q_off, kv_off, causal);
    if (ws < 0) {
      rc = g_attn(q->const_data_ptr(), k->const_data_ptr(), w->const_data_ptr(), o.mutable_data_ptr(),
                  lse.mutable_data_ptr(), b, sq, skv, hq, hkv, q_off, kv_off, causal, scale, status,
                  current_stream());
    } else {
      at::Tensor buf;
      if (ws > 0) buf = empty(*q, {ws}, at::kByte);
      rc = g_split(q->const_data_ptr(), k->const_data_ptr(), w->const_data_ptr(), o.mutable_data_ptr(),
                   lse.mutable_data_ptr(), b, sq, skv, hq, hkv, q_off, kv_off, causal, scale,
                   ws > 0 ? buf.mutable_data_ptr() : nullptr, ws, status, current_stream());
    }
  }
  if (rc == 0) {
    PyObject* t = PyTuple_New(2);
    if (t == nullptr) return nullptr;
    PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(o));
    PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(lse));
    return t;
  }
  CB_END
}

// bind({name: address}): the C entry points, from the loaded library.
PyObject* fast_bind(PyObject*, PyObject* d) {
  const auto get = [&](const char* name) -> void* {
    PyObject* o = PyDict_GetItemString(d, name);
    return o == nullptr ? nullptr : PyLong_AsVoidPtr(o);
  };
  g_gemm_bf16 = reinterpret_cast<GemmFn>(get("cb_gemm_bf16"));
  g_gemm_fp8 = reinterpret_cast<GemmFn>(get("cb_gemm_fp8"));
  g_gemm_bs = reinterpret_cast<ScaledGemmFn>(get("cb_gemm_fp8_blockscaled"));
  g_gemm_mx = reinterpret_cast<MxGemmFn>(get("cb_gemm_fp8_mx"));
  g_quant = reinterpret_cast<QuantFn>(get("cb_quant_blockscaled"));
  g_quant_pow2 = reinterpret_cast<QuantPow2Fn>(get("cb_quant_blockscaled_pow2"));
  g_attn = reinterpret_cast<AttnFn>(get("cb_attn_fwd4"));
  g_split_bytes = reinterpret_cast<SplitBytesFn>(get("cb_attn_split_bytes"));
  g_split = reinterpret_cast<SplitFn>(get("cb_attn_split"));
  if (PyErr_Occurred()) return nullptr;
  if (!g_gemm_bf16 || !g_gemm_fp8 || !g_gemm_bs || !g_gemm_mx || !g_quant || !g_quant_pow2 || !g_attn ||
      !g_split_bytes || !g_split) {
    PyErr_SetString(PyExc_RuntimeError, "fast_ops.bind: an entry point is missing");
    return nullptr;
  }
  Py_RETURN_NONE;
}

// built_for(): the PyTorch and Python whose headers this file was compiled with; asked before anything else.
PyObject* fast_built_for(PyObject*, PyObject*) { return PyUnicode_FromString(CB_BUILT_FOR); }

PyMethodDef methods[] = {
    {"built_for", fast_built_for, METH_NOARGS, nullptr},
    {"bind", fast_bind, METH_O, nullptr},
    {"gemm", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(fast_gemm)), METH_FASTCALL, nullptr},
    {"gemm_fp8_mx", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(fast_gemm_mx)), METH_FASTCALL, nullptr},
    {"gemm_fp8_blockscaled", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(fast_gemm_bs)), METH_FASTCALL,
     nullptr},
    {"quantize_rows", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(fast_quantize_rows)), METH_FASTCALL,
     nullptr},
    {"attention", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(fast_attention)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fast_ops", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fast_ops() { return PyModule_Create(&module); }
