// Host side of the operator surface: kernelforge._host, a CPython extension that takes torch tensors, checks them,
// allocates the result and calls the C ABI of libkfb200.so (include/kfb200.h).
//
// Why it is native: a small call (INT4 linear at M = 1, one decode step of attention) is 4-8 us of GPU time, while the
// same steps written in Python (validators, torch.empty, the device guard, a ctypes call with 10-18 converted
// arguments) took 15-30 us of host time per call, so the GPU waited for the host.  Here a call costs 2-4 us.
//
// Contract with kernelforge/ops.py and quantize.py: a function returns None when the call is not a plain one (a tensor
// subclass, another dtype or device, a shape the validators reject, an empty dimension).  The Python layer then runs its
// validators, which raise the documented exceptions, or takes the general route.  Nothing is cached between calls; the
// workspace of a call comes from torch's caching allocator, so streams and threads behave as for any torch tensor.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/GradMode.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>

#include "../../include/kfb200.h"

namespace {

// A plain torch.Tensor (or nn.Parameter) on a CUDA device: what the kernels take without further questions.  The wrappers of
// torch.func (vmap, grad, jvp) have the type of a plain tensor, but no memory of their own.
inline const at::Tensor* plain(PyObject* o) {
  if (!THPVariable_CheckTypeExact(Py_TYPE(o))) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  constexpr c10::DispatchKeySet wrappers({c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper});
  return t.is_cuda() && t.layout() == at::kStrided && !t.key_set().has_any(wrappers) ? &t : nullptr;
}

// Whether a tensor is being differentiated, in either mode.
inline bool differentiated(const at::Tensor& t) { return (t.requires_grad() && c10::GradMode::is_enabled()) || t._fw_grad(0).defined(); }

inline bool int_arg(PyObject* o, long long* out) {
  *out = PyLong_AsLongLong(o);
  if (*out == -1 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  return true;
}

// status code of the C ABI -> the exception kernelforge._capi.check raises for it
PyObject* raise_status(int rc) {
  if (rc == KFB_ERR_INVALID || rc == KFB_ERR_ALIGNMENT) PyErr_SetString(PyExc_ValueError, kfb_last_error());
  else PyErr_Format(PyExc_RuntimeError, "kfb200 error %d: %s", rc, kfb_last_error());
  return nullptr;
}

inline at::Tensor new_tensor(at::IntArrayRef size, at::ScalarType type, const at::Tensor& like) {
  return at::Tensor(at::detail::empty_cuda(size, type, like.device(), std::nullopt));
}

// The C ABI launches on the current device: switch to the tensors' device for the call when it is another one.
struct OnDevice {
  int prev = -1;
  explicit OnDevice(const at::Tensor& t) {
    const int want = t.device().index(), cur = c10::cuda::current_device();
    if (want != cur) {
      prev = cur;
      c10::cuda::set_device((c10::DeviceIndex)want);
    }
  }
  ~OnDevice() {
    if (prev >= 0) c10::cuda::set_device((c10::DeviceIndex)prev);
  }
};
inline void* stream_of(const at::Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// C++ exceptions become the Python ones that torch's own functions raise (torch.OutOfMemoryError and so on).
template <class F>
PyObject* guarded(F&& body) {
  HANDLE_TH_ERRORS
  return body();
  END_HANDLE_TH_ERRORS
}

// The interpreter lock is free while this lives.  An exception that passes through takes it back first (data_ptr() throws).
struct NoGil {
  PyThreadState* state = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(state); }
};

PyObject* pair_of(at::Tensor first, PyObject* second /* new reference or null */) {
  PyObject* f = second ? THPVariable_Wrap(std::move(first)) : nullptr;
  PyObject* both = f ? PyTuple_Pack(2, f, second) : nullptr;
  Py_XDECREF(f);
  Py_XDECREF(second);
  return both;
}

#define NOT_PLAIN Py_RETURN_NONE
#define ARGS(count)                                                                         \
  if (n != (count)) {                                                                       \
    PyErr_Format(PyExc_TypeError, "expected %d arguments, got %zd", (int)(count), n);       \
    return nullptr;                                                                         \
  }

inline int dtype_code(at::ScalarType t) { return t == at::kHalf ? KFB_F16 : t == at::kBFloat16 ? KFB_BF16 : t == at::kFloat ? KFB_F32 : -1; }

// int4_linear(x, packed, scales, group_size, bias or None) -> y
// int4_linear(x, packed, scales, group_size, "silu_pairs") -> silu(gate) * up for gate / up-interleaved weight rows
PyObject* int4_linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  ARGS(5)
  return guarded([&]() -> PyObject* {
    const at::Tensor *x = plain(a[0]), *packed = plain(a[1]), *scales = plain(a[2]), *bias = nullptr;
    long long group;
    if (!x || !packed || !scales || !int_arg(a[3], &group)) NOT_PLAIN;
    const auto type = x->scalar_type();
    if ((type != at::kHalf && type != at::kBFloat16) || packed->scalar_type() != at::kInt || scales->scalar_type() != at::kHalf) NOT_PLAIN;
    const bool silu = PyUnicode_Check(a[4]);
    if (a[4] != Py_None && !silu) {
      bias = plain(a[4]);
      if (!bias || differentiated(*bias)) NOT_PLAIN;   // (`y + bias` in Python then)
      if (bias->scalar_type() != type || bias->dim() != 1 || !bias->is_contiguous() || bias->device() != x->device()) NOT_PLAIN;
    }
    if (x->dim() < 1 || packed->dim() != 2 || scales->dim() != 2 || !x->is_contiguous() || !packed->is_contiguous() || !scales->is_contiguous()) NOT_PLAIN;
    if (packed->device() != x->device() || scales->device() != x->device()) NOT_PLAIN;
    const int64_t k = x->size(-1), rows = packed->size(0);
    if ((group != 64 && group != 128) || k < group || k % group || packed->size(1) * 8 != k || scales->size(0) != rows || scales->size(1) != k / group) NOT_PLAIN;
    const int64_t m = x->numel() / k;
    if (m < 1 || rows < 1 || m > INT32_MAX || rows > INT32_MAX || k > INT32_MAX || (bias && bias->size(0) != rows)) NOT_PLAIN;
    if (silu && (type != at::kHalf || rows % 4)) NOT_PLAIN;
    OnDevice dev(*x);
    at::DimVector shape(x->sizes());
    shape.back() = silu ? rows / 2 : rows;
    at::Tensor y = new_tensor(shape, type, *x);
    const int code = dtype_code(type);
    const size_t ws_bytes = kfb_int4_linear_ws_bytes((int)m, (int)rows, (int)k, (int)group, code);
    at::Tensor ws;
    if (ws_bytes) ws = new_tensor({(int64_t)ws_bytes}, at::kByte, *x);
    void *stream = stream_of(*x), *wsp = ws_bytes ? ws.data_ptr() : nullptr;
    int rc;
    {
      NoGil free;
      if (silu) rc = kfb_int4_linear_silu_pairs(x->data_ptr(), packed->data_ptr(), scales->data_ptr(), y.data_ptr(), (int)m, (int)rows, (int)k,
                                                (int)group, wsp, ws_bytes, stream);
      else rc = kfb_int4_linear(x->data_ptr(), packed->data_ptr(), scales->data_ptr(), bias ? bias->data_ptr() : nullptr, y.data_ptr(), (int)m,
                                (int)rows, (int)k, (int)group, code, wsp, ws_bytes, stream);
    }
    return rc ? raise_status(rc) : THPVariable_Wrap(std::move(y));
  });
}

// plain_constant(t) -> whether t may go into a kernel as a bias: a plain CUDA tensor outside autograd and torch.func
PyObject* plain_constant(PyObject*, PyObject* const* a, Py_ssize_t n) {
  ARGS(1)
  return guarded([&]() -> PyObject* {
    const at::Tensor* t = plain(a[0]);
    return PyBool_FromLong(t && !differentiated(*t));
  });
}

struct Attention {
  const at::Tensor *q, *k, *v;
  int64_t b, h, nq, d, hk, nk;
  int64_t strides[3];
  bool strided;   // k and v are views that the kernels read in place through `strides`
};

// The checks of ops._check_attn.  `views`: k and v may be strided (dense D axis, equal strides, multiples of 8).
bool attention_args(PyObject* const* a, bool views, Attention* p) {
  p->q = plain(a[0]); p->k = plain(a[1]); p->v = plain(a[2]);
  if (!p->q || !p->k || !p->v) return false;
  const at::Tensor &q = *p->q, &k = *p->k, &v = *p->v;
  const auto type = q.scalar_type();
  if ((type != at::kHalf && type != at::kBFloat16) || k.scalar_type() != type || v.scalar_type() != type) return false;
  if (q.dim() != 4 || k.dim() != 4 || v.dim() != 4 || k.sizes() != v.sizes() || !q.is_contiguous()) return false;
  if (k.device() != q.device() || v.device() != q.device()) return false;
  p->b = q.size(0); p->h = q.size(1); p->nq = q.size(2); p->d = q.size(3); p->hk = k.size(1); p->nk = k.size(2);
  if (k.size(0) != p->b || k.size(3) != p->d || (p->d != 64 && p->d != 128)) return false;
  if (p->b < 1 || p->h < 1 || p->nq < 1 || p->hk < 1 || p->nk < 1 || p->h % p->hk) return false;
  if (p->b > INT32_MAX || p->h > INT32_MAX || p->nq > INT32_MAX || p->nk > INT32_MAX) return false;
  p->strided = !(k.is_contiguous() && v.is_contiguous());
  if (!p->strided) return true;
  if (!views || k.strides() != v.strides() || k.stride(3) != 1) return false;
  for (int i = 0; i < 3; ++i) {
    p->strides[i] = k.stride(i);
    if (p->strides[i] % 8) return false;
  }
  return true;
}

bool scale_arg(PyObject* o, int64_t d, float* scale) {
  if (o == Py_None) {
    *scale = (float)(1.0 / std::sqrt((double)d));
    return true;
  }
  const double s = PyFloat_AsDouble(o);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  *scale = (float)s;
  return s > 0;
}

// flash_attn(q, k, v, causal, scale or None, views) -> o
PyObject* flash_attn(PyObject*, PyObject* const* a, Py_ssize_t n) {
  ARGS(6)
  return guarded([&]() -> PyObject* {
    Attention p;
    float scale;
    const int causal = PyObject_IsTrue(a[3]), views = PyObject_IsTrue(a[5]);
    if (causal < 0 || views < 0) return nullptr;
    if (!attention_args(a, views != 0, &p) || !scale_arg(a[4], p.d, &scale) || (causal && p.nq > p.nk)) NOT_PLAIN;
    OnDevice dev(*p.q);
    at::Tensor o = new_tensor(p.q->sizes(), p.q->scalar_type(), *p.q);
    const size_t ws_bytes = kfb_flash_attn_ws_bytes((int)p.b, (int)p.h, (int)p.hk, (int)p.nq, (int)p.nk, (int)p.d);
    at::Tensor ws;
    if (ws_bytes) ws = new_tensor({(int64_t)ws_bytes}, at::kByte, *p.q);
    void* stream = stream_of(*p.q);
    int rc;
    {
      NoGil free;
      rc = kfb_flash_attn_fwd(p.q->data_ptr(), p.k->data_ptr(), p.v->data_ptr(), o.data_ptr(), dtype_code(p.q->scalar_type()), (int)p.b, (int)p.h,
                              (int)p.hk, (int)p.nq, (int)p.nk, (int)p.d, causal, scale, p.strided ? p.strides : nullptr,
                              ws_bytes ? ws.data_ptr() : nullptr, ws_bytes, stream);
    }
    return rc ? raise_status(rc) : THPVariable_Wrap(std::move(o));
  });
}

// flash_attn_decode(q, k_cache, v_cache, kv_len, scale or None) -> o, and flash_attn_decode_step with the same arguments
template <decltype(&kfb_flash_attn_decode_kvlen) Entry>
PyObject* flash_attn_decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  ARGS(5)
  return guarded([&]() -> PyObject* {
    Attention p;
    float scale;
    const at::Tensor* len = plain(a[3]);
    if (!attention_args(a, true, &p) || p.nq != 1 || !scale_arg(a[4], p.d, &scale)) NOT_PLAIN;
    if (!len || len->scalar_type() != at::kInt || len->numel() != p.b || !len->is_contiguous() || len->device() != p.q->device()) NOT_PLAIN;
    OnDevice dev(*p.q);
    at::Tensor o = new_tensor(p.q->sizes(), p.q->scalar_type(), *p.q);
    const size_t ws_bytes = kfb_flash_attn_ws_bytes((int)p.b, (int)p.h, (int)p.hk, 1, (int)p.nk, (int)p.d);
    at::Tensor ws;
    if (ws_bytes) ws = new_tensor({(int64_t)ws_bytes}, at::kByte, *p.q);
    void* stream = stream_of(*p.q);
    int rc;
    {
      NoGil free;
      rc = Entry(p.q->data_ptr(), p.k->data_ptr(), p.v->data_ptr(), o.data_ptr(), dtype_code(p.q->scalar_type()), (int)p.b, (int)p.h, (int)p.hk,
                 (int)p.nk, (int)p.d, scale, p.strided ? p.strides : nullptr, static_cast<const int32_t*>(len->data_ptr()),
                 ws_bytes ? ws.data_ptr() : nullptr, ws_bytes, stream);
    }
    return rc ? raise_status(rc) : THPVariable_Wrap(std::move(o));
  });
}

// quantize_pack(weight, group_size) -> (packed, scales)
PyObject* quantize_pack(PyObject*, PyObject* const* a, Py_ssize_t n) {
  ARGS(2)
  return guarded([&]() -> PyObject* {
    const at::Tensor* w = plain(a[0]);
    long long group;
    if (!w || !int_arg(a[1], &group) || w->dim() != 2 || !w->is_contiguous() || dtype_code(w->scalar_type()) < 0) NOT_PLAIN;
    const int64_t rows = w->size(0), k = w->size(1);
    if ((group != 64 && group != 128) || rows < 1 || k < group || k % group || rows > INT32_MAX || k > INT32_MAX) NOT_PLAIN;
    OnDevice dev(*w);
    at::Tensor packed = new_tensor({rows, k / 8}, at::kInt, *w), scales = new_tensor({rows, k / group}, at::kHalf, *w);
    void* stream = stream_of(*w);
    int rc;
    {
      NoGil free;
      rc = kfb_quantize_pack(w->data_ptr(), dtype_code(w->scalar_type()), (int)rows, (int)k, (int)group, packed.data_ptr(), scales.data_ptr(), stream);
    }
    if (rc) return raise_status(rc);
    return pair_of(std::move(packed), THPVariable_Wrap(std::move(scales)));
  });
}

// fp16, contiguous, on x's device
inline bool half_like(const at::Tensor* t, const at::Tensor& x) {
  return t && t->scalar_type() == at::kHalf && t->is_contiguous() && t->device() == x.device();
}

// add_rmsnorm(x, weight, eps, residual or None) -> (y, s): x [rows, hidden]
PyObject* add_rmsnorm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  ARGS(4)
  return guarded([&]() -> PyObject* {
    const at::Tensor *x = plain(a[0]), *w = plain(a[1]), *res = nullptr;
    const double eps = PyFloat_AsDouble(a[2]);
    if (PyErr_Occurred()) return nullptr;
    if (!x || x->dim() != 2 || !half_like(x, *x) || !half_like(w, *x) || w->numel() != x->size(1)) NOT_PLAIN;
    if (a[3] != Py_None) {
      res = plain(a[3]);
      if (!half_like(res, *x) || res->sizes() != x->sizes()) NOT_PLAIN;
    }
    OnDevice dev(*x);
    at::Tensor y = new_tensor(x->sizes(), at::kHalf, *x), s;
    if (res) s = new_tensor(x->sizes(), at::kHalf, *x);
    void* stream = stream_of(*x);
    int rc;
    {
      NoGil free;
      rc = kfb_add_rmsnorm(x->data_ptr(), res ? res->data_ptr() : nullptr, w->data_ptr(), y.data_ptr(), res ? s.data_ptr() : nullptr,
                           (int)x->size(0), (int)x->size(1), (float)eps, stream);
    }
    if (rc) return raise_status(rc);
    if (res) return pair_of(std::move(y), THPVariable_Wrap(std::move(s)));
    Py_INCREF(a[0]);
    return pair_of(std::move(y), a[0]);
  });
}

// rope_tokens(qkv, cos, sin, k_cache, v_cache, batch, heads, pairs) -> q [B, T, H, D]: qkv [B * T, (H + 2 Hk) D]
PyObject* rope_tokens(PyObject*, PyObject* const* a, Py_ssize_t n) {
  ARGS(8)
  return guarded([&]() -> PyObject* {
    const at::Tensor *qkv = plain(a[0]), *cos = plain(a[1]), *sin = plain(a[2]), *kc = plain(a[3]), *vc = plain(a[4]);
    long long b, h;
    const int pairs = PyObject_IsTrue(a[7]);
    if (!int_arg(a[5], &b) || !int_arg(a[6], &h) || pairs < 0) NOT_PLAIN;
    if (!qkv || !half_like(qkv, *qkv) || !half_like(kc, *qkv) || !half_like(vc, *qkv) || !cos || !sin) NOT_PLAIN;
    if (kc->dim() != 4 || kc->sizes() != vc->sizes() || kc->size(0) != b || b < 1 || qkv->dim() != 2 || qkv->size(0) % b) NOT_PLAIN;
    const int64_t t = qkv->size(0) / b, hk = kc->size(1), lmax = kc->size(2), d = kc->size(3);
    for (const at::Tensor* table : {cos, sin})
      if (table->scalar_type() != at::kFloat || !table->is_contiguous() || table->dim() != 2 || table->size(0) < t || table->size(1) != d ||
          table->device() != qkv->device())
        NOT_PLAIN;
    if (qkv->size(1) != (h + 2 * hk) * d) NOT_PLAIN;
    OnDevice dev(*qkv);
    at::Tensor q = new_tensor({b, t, h, d}, at::kHalf, *qkv);
    void* stream = stream_of(*qkv);
    int rc;
    {
      NoGil free;
      rc = kfb_rope_tokens(qkv->data_ptr(), cos->data_ptr(), sin->data_ptr(), q.data_ptr(), kc->data_ptr(), vc->data_ptr(), (int)b, (int)t, (int)h,
                           (int)hk, (int)d, (int)lmax, pairs, stream);
    }
    return rc ? raise_status(rc) : THPVariable_Wrap(std::move(q));
  });
}

// attention_tokens(q, k_cache, v_cache, kv_rows, causal) -> o: q and o [B, T, H, D], the first kv_rows rows of the caches
PyObject* attention_tokens(PyObject*, PyObject* const* a, Py_ssize_t n) {
  ARGS(5)
  return guarded([&]() -> PyObject* {
    const at::Tensor *q = plain(a[0]), *kc = plain(a[1]), *vc = plain(a[2]);
    long long nk;
    const int causal = PyObject_IsTrue(a[4]);
    if (!int_arg(a[3], &nk) || causal < 0) NOT_PLAIN;
    if (!q || q->dim() != 4 || !half_like(q, *q) || !half_like(kc, *q) || !half_like(vc, *q) || kc->dim() != 4 || kc->sizes() != vc->sizes()) NOT_PLAIN;
    const int64_t b = q->size(0), t = q->size(1), h = q->size(2), d = q->size(3), hk = kc->size(1), lmax = kc->size(2);
    if (kc->size(0) != b || kc->size(3) != d || nk < 1 || nk > lmax || t < 1) NOT_PLAIN;
    const int64_t strides[3] = {hk * lmax * d, lmax * d, d};
    OnDevice dev(*q);
    at::Tensor o = new_tensor(q->sizes(), at::kHalf, *q);
    const size_t ws_bytes = kfb_flash_attn_ws_bytes((int)b, (int)h, (int)hk, (int)t, (int)nk, (int)d);
    at::Tensor ws;
    if (ws_bytes) ws = new_tensor({(int64_t)ws_bytes}, at::kByte, *q);
    void* stream = stream_of(*q);
    int rc;
    {
      NoGil free;
      rc = kfb_flash_attn_fwd_tokens(q->data_ptr(), kc->data_ptr(), vc->data_ptr(), o.data_ptr(), KFB_F16, (int)b, (int)h, (int)hk, (int)t, (int)nk,
                                     (int)d, causal, (float)(1.0 / std::sqrt((double)d)), strides, ws_bytes ? ws.data_ptr() : nullptr, ws_bytes, stream);
    }
    return rc ? raise_status(rc) : THPVariable_Wrap(std::move(o));
  });
}

// silu_mul(gate_up, pairs) -> act [rows, inter]: gate_up [rows, 2 * inter], gate | up or (pairs) side by side
PyObject* silu_mul(PyObject*, PyObject* const* a, Py_ssize_t n) {
  ARGS(2)
  return guarded([&]() -> PyObject* {
    const at::Tensor* gu = plain(a[0]);
    const int pairs = PyObject_IsTrue(a[1]);
    if (pairs < 0 || !gu || gu->dim() != 2 || !half_like(gu, *gu) || gu->size(1) % 2) NOT_PLAIN;
    const int64_t rows = gu->size(0), inter = gu->size(1) / 2;
    OnDevice dev(*gu);
    at::Tensor act = new_tensor({rows, inter}, at::kHalf, *gu);
    void* stream = stream_of(*gu);
    int rc;
    {
      NoGil free;
      rc = pairs ? kfb_silu_mul_pairs(gu->data_ptr(), act.data_ptr(), (int)rows, (int)inter, stream)
                 : kfb_silu_mul(gu->data_ptr(), act.data_ptr(), (int)rows, (int)inter, stream);
    }
    return rc ? raise_status(rc) : THPVariable_Wrap(std::move(act));
  });
}

#define METHOD(name, doc) {#name, (PyCFunction)(void*)name, METH_FASTCALL, doc}
PyMethodDef methods[] = {
    METHOD(int4_linear, "int4_linear(x, packed, scales, group_size, bias) -> y, or None when the call is not a plain one"),
    METHOD(plain_constant, "plain_constant(t) -> whether t may go into a kernel as a bias"),
    METHOD(flash_attn, "flash_attn(q, k, v, causal, scale, views) -> o, or None when the call is not a plain one"),
    {"flash_attn_decode", (PyCFunction)(void*)flash_attn_decode<kfb_flash_attn_decode_kvlen>, METH_FASTCALL,
     "flash_attn_decode(q, k_cache, v_cache, kv_len, scale) -> o, or None when the call is not a plain one"},
    {"flash_attn_decode_step", (PyCFunction)(void*)flash_attn_decode<kfb_flash_attn_decode_step>, METH_FASTCALL,
     "flash_attn_decode_step(q, k_cache, v_cache, kv_len, scale) -> o, or None when the call is not a plain one"},
    METHOD(quantize_pack, "quantize_pack(weight, group_size) -> (packed, scales), or None when the call is not a plain one"),
    METHOD(add_rmsnorm, "add_rmsnorm(x, weight, eps, residual) -> (y, s), or None"),
    METHOD(rope_tokens, "rope_tokens(qkv, cos, sin, k_cache, v_cache, batch, heads, pairs) -> q [B, T, H, D], or None"),
    METHOD(attention_tokens, "attention_tokens(q, k_cache, v_cache, kv_rows, causal) -> o [B, T, H, D], or None"),
    METHOD(silu_mul, "silu_mul(gate_up, pairs) -> act, or None"),
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "Checked, allocating calls of libkfb200.so on torch tensors.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) { return PyModule_Create(&module); }
