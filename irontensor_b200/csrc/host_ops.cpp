// The host side of the ops, natively: argument checks, output and workspace allocation, and the C-ABI call, in one step from
// Python.  A small attention call spends 7 to 30 us on the GPU; the same steps in Python over ctypes took 30 to 140 us, so the
// GPU waited for the host on every launch-bound shape.
//
// TensorBase is the storage behind irontensor_b200.Tensor: one torch tensor of the logical shape (device memory comes from
// torch's caching allocator, on the current stream) and the optional `lse` side output.  Every op function here takes the plain
// case -- packed tensors on the current device, shapes and precisions that fit together, nothing empty -- and returns None otherwise:
// the Python function of the same name then raises the reference's assertion, or handles the case.
// Workspaces are allocated per call (stream-ordered reuse is the allocator's), so calls on different streams or threads share
// nothing.  The GIL is released around the C-ABI calls.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <structmember.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <new>
#include <vector>

#include "../../include/irontensor_b200.h"

namespace {

struct TensorObject {
  PyObject_HEAD
  at::Tensor t;
  PyObject* lse;
};

PyTypeObject* g_base = nullptr;      // TensorBase
PyTypeObject* g_tensor = nullptr;    // irontensor_b200.Tensor, what the ops return
PyObject* g_fp32 = nullptr;          // Precision.FP32 / .BF16
PyObject* g_bf16 = nullptr;
PyObject* g_check = nullptr;         // status -> exception
PyObject* g_context = nullptr;       // device -> _Context

struct Device {
  it_ctx* ctx = nullptr;
  std::vector<std::pair<cudaStream_t, it_stream*>> streams;
};
Device g_devices[64];                // guarded by the GIL

at::Tensor& ten(PyObject* o) { return reinterpret_cast<TensorObject*>(o)->t; }
bool is_tensor(PyObject* o) { return PyObject_TypeCheck(o, g_base) && ten(o).defined(); }
bool is_bf16(const at::Tensor& t) { return t.scalar_type() == at::kBFloat16; }

PyObject* wrap(at::Tensor&& t) {
  PyObject* o = g_tensor->tp_alloc(g_tensor, 0);
  if (o == nullptr) return nullptr;
  new (&ten(o)) at::Tensor(std::move(t));
  reinterpret_cast<TensorObject*>(o)->lse = nullptr;
  return o;
}
PyObject* wrap_with_lse(at::Tensor&& t, at::Tensor&& lse) {
  PyObject* l = wrap(std::move(lse));
  if (l == nullptr) return nullptr;
  PyObject* o = wrap(std::move(t));
  if (o == nullptr) {
    Py_DECREF(l);
    return nullptr;
  }
  reinterpret_cast<TensorObject*>(o)->lse = l;
  return o;
}
PyObject* wrap_tuple(at::Tensor* t, int n) {
  PyObject* r = PyTuple_New(n);
  for (int i = 0; r != nullptr && i < n; ++i) {
    PyObject* o = wrap(std::move(t[i]));
    if (o == nullptr) Py_CLEAR(r);
    else PyTuple_SET_ITEM(r, i, o);
  }
  return r;
}

// The library's context of the current device and its object for torch's current stream.  False with an exception set.
struct Where {
  int device;
  it_ctx* ctx;
  it_stream* stream;
};
PyObject* ctx_object(int device) { return PyObject_CallFunction(g_context, "i", device); }
uintptr_t handle_of(PyObject* c_void_p) {   // ctypes.c_void_p -> address
  PyObject* v = PyObject_GetAttrString(c_void_p, "value");
  const uintptr_t a = v != nullptr ? reinterpret_cast<uintptr_t>(PyLong_AsVoidPtr(v)) : 0;
  Py_XDECREF(v);
  return a;
}
bool where(Where* w) {
  w->device = c10::cuda::current_device();
  const cudaStream_t s = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(w->device)).stream();
  Device& d = g_devices[w->device & 63];
  w->ctx = d.ctx;
  for (const auto& e : d.streams)
    if (e.first == s) {
      w->stream = e.second;
      return true;
    }
  PyObject* c = ctx_object(w->device);   // first call on this device or stream: the Python context object owns both handles
  if (c == nullptr) return false;
  PyObject* h = PyObject_GetAttrString(c, "handle");
  PyObject* st = h != nullptr ? PyObject_CallMethod(c, "stream", nullptr) : nullptr;
  bool ok = st != nullptr;
  if (ok) {
    d.ctx = w->ctx = reinterpret_cast<it_ctx*>(handle_of(h));
    w->stream = reinterpret_cast<it_stream*>(handle_of(st));
    ok = !PyErr_Occurred() && w->ctx != nullptr && w->stream != nullptr;
    if (ok) d.streams.emplace_back(s, w->stream);
  }
  Py_XDECREF(st);
  Py_XDECREF(h);
  Py_DECREF(c);
  return ok;
}

at::Tensor empty(const Where& w, at::IntArrayRef shape, at::ScalarType type) {
  return at::detail::empty_cuda(shape, type, c10::Device(c10::DeviceType::CUDA, static_cast<c10::DeviceIndex>(w.device)), std::nullopt);
}
at::Tensor scratch(const Where& w, size_t bytes) { return empty(w, {static_cast<int64_t>(bytes)}, at::kByte); }

bool raise_status(it_status rc) {   // true: no error
  if (rc == IT_OK) return true;
  PyObject* r = PyObject_CallFunction(g_check, "i", static_cast<int>(rc));
  if (r != nullptr) {
    Py_DECREF(r);
    PyErr_SetString(PyExc_RuntimeError, "irontensor_b200: call failed");
  }
  return false;
}
template <typename F>
bool call(F&& f) {
  it_status rc;
  Py_BEGIN_ALLOW_THREADS
  rc = f();
  Py_END_ALLOW_THREADS
  return raise_status(rc);
}

// The plain case: a contiguous, non-empty fp32 or bf16 tensor of `dim` dimensions on the current device.
bool plain(PyObject* o, int64_t dim) {
  if (!is_tensor(o)) return false;
  const at::Tensor& t = ten(o);
  return (is_bf16(t) || t.scalar_type() == at::kFloat) && t.dim() == dim && t.is_cuda() && t.numel() > 0 && t.is_contiguous() &&
         t.get_device() == c10::cuda::current_device();
}
bool same(const at::Tensor& a, const at::Tensor& b) { return a.sizes() == b.sizes() && a.scalar_type() == b.scalar_type(); }
it_dtype dtype_of(const at::Tensor& t) { return is_bf16(t) ? IT_BF16 : IT_F32; }

// Plain numbers and truth values of 32 bits; false, without an exception, for anything else, which the Python function then
// converts or refuses.
bool as_int(PyObject* o, int32_t* v) {
  if (!PyIndex_Check(o)) return false;
  const Py_ssize_t x = PyNumber_AsSsize_t(o, nullptr);   // out of range: clipped
  if (x == -1 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  *v = static_cast<int32_t>(x);
  return *v == x;
}
bool as_float(PyObject* o, float* v) {
  if (!PyFloat_Check(o) && !PyLong_Check(o)) return false;
  const double x = PyFloat_AsDouble(o);
  if (x == -1.0 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  *v = static_cast<float>(x);
  return true;
}
bool as_bool(PyObject* o, int32_t* v) {
  if (!PyLong_Check(o)) return false;
  *v = PyObject_IsTrue(o);
  return true;
}

#define IT_ARGS(n)                                                                                    \
  if (nargs != (n)) {                                                                                 \
    PyErr_Format(PyExc_TypeError, "%s takes %d arguments, got %zd", __func__, (n), nargs);            \
    return nullptr;                                                                                   \
  }
template <typename F>
PyObject* guard(F&& f) {   // C++ exceptions as Python's
  try {
    return f();
  } catch (...) {   // as torch's own functions report them: torch.OutOfMemoryError from the allocator, RuntimeError, ...
    if (!PyErr_Occurred()) torch::translate_exception_to_python(std::current_exception());
    return nullptr;
  }
}

// ------------------------------------------------------------------------------------------------ attention
// q, k, v, causal.  BHSD: [batch, heads, seq, head_dim], one shape.  Otherwise [batch, seq, heads, head_dim], k and v with a
// number of heads that divides q's (`grouped`) or q's own.
template <bool BHSD>
PyObject* attention_fwd(PyObject* const* a, bool grouped) {
  return guard([&]() -> PyObject* {
    if (!plain(a[0], 4) || !plain(a[1], 4) || !plain(a[2], 4)) Py_RETURN_NONE;
    const at::Tensor &q = ten(a[0]), &k = ten(a[1]), &v = ten(a[2]);
    if (!same(k, v) || q.scalar_type() != k.scalar_type() || q.size(3) > 128) Py_RETURN_NONE;
    const int64_t B = q.size(0), S = q.size(BHSD ? 2 : 1), H = q.size(BHSD ? 1 : 2), D = q.size(3);
    int64_t Hkv = H;
    if (!grouped) {
      if (q.sizes() != k.sizes()) Py_RETURN_NONE;
    } else {
      Hkv = k.size(2);
      if (k.size(0) != B || k.size(1) != S || k.size(3) != D || H % Hkv != 0) Py_RETURN_NONE;
    }
    int32_t causal;
    Where w;
    if (!as_bool(a[3], &causal)) Py_RETURN_NONE;
    if (!where(&w)) return nullptr;
    at::Tensor o = empty(w, q.sizes(), q.scalar_type()), lse = empty(w, {B, H, S}, at::kFloat);
    const void *pq = q.data_ptr(), *pk = k.data_ptr(), *pv = v.data_ptr();
    void* po = o.data_ptr();
    float* pl = lse.data_ptr<float>();
    const it_dtype dt = dtype_of(q);
    if (!call([&] {
          return BHSD ? it_flash_attention_fwd(w.ctx, w.stream, dt, B, H, S, D, causal, pq, pk, pv, po, pl)
                      : it_attention_gqa_fwd(w.ctx, w.stream, dt, B, S, H, Hkv, D, causal, pq, pk, pv, po, pl);
        }))
      return nullptr;
    return wrap_with_lse(std::move(o), std::move(lse));
  });
}
PyObject* flash_attention(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  IT_ARGS(4);
  return attention_fwd<true>(a, false);
}
PyObject* attention(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  IT_ARGS(4);
  return attention_fwd<false>(a, false);
}
PyObject* attention_gqa(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  IT_ARGS(4);
  return attention_fwd<false>(a, true);
}

// grad_output, q, k, v, o, lse, causal, rope_base (None: no rotation), position_offset
template <bool BHSD>
PyObject* attention_bwd(PyObject* const* a, bool grouped) {
  return guard([&]() -> PyObject* {
    for (int i = 0; i < 5; ++i)
      if (!plain(a[i], 4)) Py_RETURN_NONE;
    if (!plain(a[5], 3)) Py_RETURN_NONE;
    const at::Tensor &g = ten(a[0]), &q = ten(a[1]), &k = ten(a[2]), &v = ten(a[3]), &o = ten(a[4]), &lse = ten(a[5]);
    if (!same(g, q) || !same(o, q) || !same(k, v) || q.scalar_type() != k.scalar_type() || lse.scalar_type() != at::kFloat ||
        q.size(3) > 128)
      Py_RETURN_NONE;
    const int64_t B = q.size(0), S = q.size(BHSD ? 2 : 1), H = q.size(BHSD ? 1 : 2), D = q.size(3);
    if (lse.numel() != B * H * S) Py_RETURN_NONE;
    int64_t Hkv = H;
    if (!grouped) {
      if (q.sizes() != k.sizes()) Py_RETURN_NONE;
    } else {
      Hkv = k.size(2);
      if (k.size(0) != B || k.size(1) != S || k.size(3) != D || H % Hkv != 0) Py_RETURN_NONE;
    }
    int32_t causal, pos = 0;
    float base = 0.f;
    const bool rope = a[7] != Py_None;
    Where w;
    if (!as_bool(a[6], &causal) || (rope && (!as_float(a[7], &base) || !as_int(a[8], &pos)))) Py_RETURN_NONE;
    if (!where(&w)) return nullptr;
    const it_dtype dt = dtype_of(q);
    size_t ws_bytes = 0;
    if (!raise_status(it_flash_attention_bwd_workspace_bytes(dt, B, H, S, D, &ws_bytes))) return nullptr;
    at::Tensor out[3] = {empty(w, q.sizes(), q.scalar_type()), empty(w, k.sizes(), k.scalar_type()), empty(w, v.sizes(), v.scalar_type())};
    at::Tensor ws = scratch(w, ws_bytes);
    const void *pg = g.data_ptr(), *pq = q.data_ptr(), *pk = k.data_ptr(), *pv = v.data_ptr(), *po = o.data_ptr();
    const float* pl = lse.data_ptr<float>();
    void *dq = out[0].data_ptr(), *dk = out[1].data_ptr(), *dv = out[2].data_ptr(), *pw = ws.data_ptr();
    if (!call([&] {
          if (BHSD) return it_flash_attention_bwd(w.ctx, w.stream, dt, B, H, S, D, causal, pq, pk, pv, po, pg, pl, dq, dk, dv, pw, ws_bytes);
          if (rope)
            return it_attention_gqa_bwd_rope(w.ctx, w.stream, dt, B, S, H, Hkv, D, causal, base, pos, pq, pk, pv, po, pg, pl, dq, dk, dv,
                                             pw, ws_bytes);
          return it_attention_gqa_bwd(w.ctx, w.stream, dt, B, S, H, Hkv, D, causal, pq, pk, pv, po, pg, pl, dq, dk, dv, pw, ws_bytes);
        }))
      return nullptr;
    return wrap_tuple(out, 3);
  });
}
PyObject* attention_backward_recompute(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  IT_ARGS(7);
  PyObject* const b[9] = {a[0], a[1], a[2], a[3], a[4], a[5], a[6], Py_None, Py_None};
  return attention_bwd<true>(b, false);
}
PyObject* attention_gqa_backward(PyObject*, PyObject* const* a, Py_ssize_t nargs) {   // grad, q, k, v, o, causal, base, offset
  IT_ARGS(8);
  if (!is_tensor(a[4]) || reinterpret_cast<TensorObject*>(a[4])->lse == nullptr) Py_RETURN_NONE;
  PyObject* const b[9] = {a[0], a[1], a[2], a[3], a[4], reinterpret_cast<TensorObject*>(a[4])->lse, a[5], a[6], a[7]};
  return attention_bwd<false>(b, true);
}
PyObject* attention_backward(PyObject*, PyObject* const* a, Py_ssize_t nargs) {   // grad, q, k, v, o, causal
  IT_ARGS(6);
  if (!is_tensor(a[4]) || reinterpret_cast<TensorObject*>(a[4])->lse == nullptr) Py_RETURN_NONE;
  PyObject* const b[9] = {a[0], a[1], a[2], a[3], a[4], reinterpret_cast<TensorObject*>(a[4])->lse, a[5], Py_None, Py_None};
  return attention_bwd<false>(b, false);
}

// q [batch, heads, head_dim], k_cache, v_cache [batch, max_len, kv_heads, head_dim], kv_len
PyObject* attention_decode(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  IT_ARGS(4);
  return guard([&]() -> PyObject* {
    if (!plain(a[0], 3) || !plain(a[1], 4) || !plain(a[2], 4)) Py_RETURN_NONE;
    const at::Tensor &q = ten(a[0]), &k = ten(a[1]), &v = ten(a[2]);
    const int64_t B = q.size(0), H = q.size(1), D = q.size(2), max_len = k.size(1), Hkv = k.size(2);
    if (!same(k, v) || q.scalar_type() != k.scalar_type() || k.size(0) != B || k.size(3) != D || H % Hkv != 0 || D > 128) Py_RETURN_NONE;
    int32_t kv_len;
    if (!as_int(a[3], &kv_len) || kv_len < 1 || kv_len > max_len) Py_RETURN_NONE;
    Where w;
    if (!where(&w)) return nullptr;
    size_t ws_bytes = 0;
    if (!raise_status(it_attention_decode_workspace_bytes(B, H, D, &ws_bytes))) return nullptr;
    at::Tensor o = empty(w, q.sizes(), q.scalar_type()), lse = empty(w, {B, H}, at::kFloat), ws = scratch(w, ws_bytes);
    const void *pq = q.data_ptr(), *pk = k.data_ptr(), *pv = v.data_ptr();
    void *po = o.data_ptr(), *pw = ws.data_ptr();
    float* pl = lse.data_ptr<float>();
    const it_dtype dt = dtype_of(q);
    if (!call([&] { return it_attention_decode(w.ctx, w.stream, dt, B, H, Hkv, D, kv_len, max_len, pq, pk, pv, po, pl, pw, ws_bytes); }))
      return nullptr;
    return wrap_with_lse(std::move(o), std::move(lse));
  });
}

// qkv [batch, seq, (heads + 2 kv_heads) * head_dim], heads, kv_heads, head_dim, causal
PyObject* attention_packed(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  IT_ARGS(5);
  return guard([&]() -> PyObject* {
    if (!plain(a[0], 3)) Py_RETURN_NONE;
    const at::Tensor& x = ten(a[0]);
    int32_t H, Hkv, D, causal;
    if (!as_int(a[1], &H) || !as_int(a[2], &Hkv) || !as_int(a[3], &D) || !as_bool(a[4], &causal)) Py_RETURN_NONE;
    const int64_t B = x.size(0), S = x.size(1);
    if (!is_bf16(x) || x.size(2) != (static_cast<int64_t>(H) + 2LL * Hkv) * D || H < 1 || Hkv < 1 || D < 1) Py_RETURN_NONE;
    Where w;
    if (!where(&w)) return nullptr;
    at::Tensor o = empty(w, {B, S, H, D}, at::kBFloat16), lse = empty(w, {B, H, S}, at::kFloat);
    const void* px = x.data_ptr();
    void* po = o.data_ptr();
    float* pl = lse.data_ptr<float>();
    if (!call([&] { return it_attention_packed_fwd(w.ctx, w.stream, IT_BF16, B, S, H, Hkv, D, causal, px, po, pl); })) return nullptr;
    return wrap_with_lse(std::move(o), std::move(lse));
  });
}

// grad_output, qkv, o, heads, kv_heads, head_dim, causal, rope_base (0: no rotation), position_offset
PyObject* attention_packed_backward(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  IT_ARGS(9);
  return guard([&]() -> PyObject* {
    if (!plain(a[0], 4) || !plain(a[1], 3) || !plain(a[2], 4)) Py_RETURN_NONE;
    PyObject* l = reinterpret_cast<TensorObject*>(a[2])->lse;
    if (l == nullptr || !plain(l, 3)) Py_RETURN_NONE;
    const at::Tensor &g = ten(a[0]), &x = ten(a[1]), &o = ten(a[2]), &lse = ten(l);
    int32_t H, Hkv, D, causal, pos;
    float base;
    if (!as_int(a[3], &H) || !as_int(a[4], &Hkv) || !as_int(a[5], &D) || !as_bool(a[6], &causal) || !as_float(a[7], &base) ||
        !as_int(a[8], &pos))
      Py_RETURN_NONE;
    const int64_t B = x.size(0), S = x.size(1);
    const int64_t want[4] = {B, S, H, D};
    if (!is_bf16(x) || !same(g, o) || !is_bf16(g) || g.sizes() != at::IntArrayRef(want, 4) || lse.numel() != B * H * S || H < 1 || Hkv < 1 ||
        D < 1 || D > 128 || x.size(2) != (static_cast<int64_t>(H) + 2LL * Hkv) * D)
      Py_RETURN_NONE;
    Where w;
    size_t ws_bytes = 0;
    if (!where(&w) || !raise_status(it_flash_attention_bwd_workspace_bytes(IT_BF16, B, H, S, D, &ws_bytes))) return nullptr;
    at::Tensor d = empty(w, x.sizes(), at::kBFloat16), ws = scratch(w, ws_bytes);
    const void *pg = g.data_ptr(), *px = x.data_ptr(), *po = o.data_ptr();
    const float* pl = lse.data_ptr<float>();
    void *pd = d.data_ptr(), *pw = ws.data_ptr();
    if (!call([&] {
          return it_attention_packed_bwd(w.ctx, w.stream, IT_BF16, B, S, H, Hkv, D, causal, base, pos, px, po, pg, pl, pd, pw, ws_bytes);
        }))
      return nullptr;
    return wrap(std::move(d));
  });
}

// ------------------------------------------------------------------------------------------------ rotary embedding
// q, k (None: q alone), base, position_offset, inverse -> (q, k) or q
PyObject* rope_qk(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  IT_ARGS(5);
  return guard([&]() -> PyObject* {
    const bool two = a[1] != Py_None;
    if (!plain(a[0], 4) || (two && !plain(a[1], 4))) Py_RETURN_NONE;
    const at::Tensor& q = ten(a[0]);
    const int64_t B = q.size(0), S = q.size(1), H = q.size(2), D = q.size(3);
    int64_t Hkv = 0;
    if (two) {
      const at::Tensor& k = ten(a[1]);
      Hkv = k.size(2);
      if (k.scalar_type() != q.scalar_type() || k.size(0) != B || k.size(1) != S || k.size(3) != D) Py_RETURN_NONE;
    }
    if (D % 2 != 0) Py_RETURN_NONE;
    float base;
    int32_t pos, inverse;
    Where w;
    if (!as_float(a[2], &base) || !as_int(a[3], &pos) || !as_bool(a[4], &inverse)) Py_RETURN_NONE;
    if (!where(&w)) return nullptr;
    at::Tensor out[2] = {empty(w, q.sizes(), q.scalar_type()), two ? empty(w, ten(a[1]).sizes(), q.scalar_type()) : at::Tensor()};
    const void *pq = q.data_ptr(), *pk = two ? ten(a[1]).data_ptr() : nullptr;
    void *oq = out[0].data_ptr(), *ok = two ? out[1].data_ptr() : nullptr;
    const it_dtype dt = dtype_of(q);
    if (!call([&] { return it_rope_qk(w.ctx, w.stream, dt, B, S, H, Hkv, D, base, pos, inverse, pq, pk, oq, ok); })) return nullptr;
    return two ? wrap_tuple(out, 2) : wrap(std::move(out[0]));
  });
}

// ------------------------------------------------------------------------------------------------ projections
PyObject* linear_forward(PyObject*, PyObject* const* a, Py_ssize_t nargs) {   // x [n, in], w [out, in]
  IT_ARGS(2);
  return guard([&]() -> PyObject* {
    if (!plain(a[0], 2) || !plain(a[1], 2)) Py_RETURN_NONE;
    const at::Tensor &x = ten(a[0]), &wt = ten(a[1]);
    if (!is_bf16(x) || !is_bf16(wt) || x.size(1) != wt.size(1)) Py_RETURN_NONE;
    const int64_t n = x.size(0), in = x.size(1), out = wt.size(0);
    Where w;
    if (!where(&w)) return nullptr;
    at::Tensor y = empty(w, {n, out}, at::kBFloat16);
    const void *px = x.data_ptr(), *pw = wt.data_ptr();
    void* py = y.data_ptr();
    if (!call([&] { return it_linear_fwd(w.ctx, w.stream, n, in, out, px, pw, py); })) return nullptr;
    return wrap(std::move(y));
  });
}

PyObject* linear_backward(PyObject*, PyObject* const* a, Py_ssize_t nargs) {   // dy [n, out], x [n, in], w [out, in]
  IT_ARGS(3);
  return guard([&]() -> PyObject* {
    if (!plain(a[0], 2) || !plain(a[1], 2) || !plain(a[2], 2)) Py_RETURN_NONE;
    const at::Tensor &dy = ten(a[0]), &x = ten(a[1]), &wt = ten(a[2]);
    const int64_t n = dy.size(0), out = dy.size(1), in = x.size(1);
    if (!is_bf16(dy) || !is_bf16(x) || !is_bf16(wt) || x.size(0) != n || wt.size(0) != out || wt.size(1) != in) Py_RETURN_NONE;
    Where w;
    if (!where(&w)) return nullptr;
    at::Tensor d[2] = {empty(w, {n, in}, at::kBFloat16), empty(w, {out, in}, at::kFloat)};
    const void *pdy = dy.data_ptr(), *px = x.data_ptr(), *pw = wt.data_ptr();
    void* dx = d[0].data_ptr();
    float* dw = d[1].data_ptr<float>();
    if (!call([&] { return it_linear_bwd(w.ctx, w.stream, n, in, out, pdy, px, pw, dx, dw); })) return nullptr;
    return wrap_tuple(d, 2);
  });
}

// x [batch, seq, hidden], w_qkv, heads, kv_heads, head_dim, rope_base (0: no rotation), position_offset, packed
PyObject* qkv_rope_forward(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  IT_ARGS(8);
  return guard([&]() -> PyObject* {
    if (!plain(a[0], 3) || !plain(a[1], 2)) Py_RETURN_NONE;
    const at::Tensor &x = ten(a[0]), &wt = ten(a[1]);
    int32_t H, Hkv, D, pos, packed;
    float base;
    if (!as_int(a[2], &H) || !as_int(a[3], &Hkv) || !as_int(a[4], &D) || !as_float(a[5], &base) || !as_int(a[6], &pos) ||
        !as_bool(a[7], &packed))
      Py_RETURN_NONE;
    const int64_t B = x.size(0), S = x.size(1), hidden = x.size(2), width = (static_cast<int64_t>(H) + 2LL * Hkv) * D;
    if (!is_bf16(x) || !is_bf16(wt) || H < 1 || Hkv < 1 || D < 2 || D > 128 || D % 2 != 0 || wt.size(0) != width || wt.size(1) != hidden)
      Py_RETURN_NONE;
    Where w;
    size_t ws_bytes = 0;
    if (!where(&w) || !raise_status(it_qkv_rope_workspace_bytes(S, D, &ws_bytes))) return nullptr;
    at::Tensor out[3];
    if (packed) {
      out[0] = empty(w, {B, S, width}, at::kBFloat16);
    } else {
      out[0] = empty(w, {B, S, H, D}, at::kBFloat16);
      out[1] = empty(w, {B, S, Hkv, D}, at::kBFloat16);
      out[2] = empty(w, {B, S, Hkv, D}, at::kBFloat16);
    }
    at::Tensor ws = scratch(w, ws_bytes);
    const void *px = x.data_ptr(), *pw = wt.data_ptr();
    void *o0 = out[0].data_ptr(), *o1 = packed ? nullptr : out[1].data_ptr(), *o2 = packed ? nullptr : out[2].data_ptr(), *pws = ws.data_ptr();
    if (!call([&] { return it_qkv_rope_fwd(w.ctx, w.stream, B, S, hidden, H, Hkv, D, base, pos, px, pw, o0, o1, o2, pws, ws_bytes); }))
      return nullptr;
    return packed ? wrap(std::move(out[0])) : wrap_tuple(out, 3);
  });
}

// ------------------------------------------------------------------------------------------------ TensorBase
PyObject* tensor_new(PyTypeObject* type, PyObject*, PyObject*) {
  PyObject* o = type->tp_alloc(type, 0);
  if (o != nullptr) {
    new (&ten(o)) at::Tensor();
    reinterpret_cast<TensorObject*>(o)->lse = nullptr;
  }
  return o;
}
void tensor_dealloc(PyObject* o) {
  ten(o).~Tensor();
  Py_CLEAR(reinterpret_cast<TensorObject*>(o)->lse);
  Py_TYPE(o)->tp_free(o);
}
int tensor_traverse(PyObject* o, visitproc visit, void* arg) {
  Py_VISIT(reinterpret_cast<TensorObject*>(o)->lse);
  return 0;
}
int tensor_clear(PyObject* o) {
  Py_CLEAR(reinterpret_cast<TensorObject*>(o)->lse);
  return 0;
}
bool read_shape(PyObject* shape, c10::SmallVector<int64_t, 6>* dims, int64_t* numel) {   // numel: -1 where 64 bits do not hold it
  PyObject* seq = PySequence_Fast(shape, "a shape is a sequence of numbers");
  if (seq == nullptr) return false;
  *numel = 1;
  bool over = false;
  for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(seq); ++i) {
    dims->push_back(PyLong_AsLongLong(PySequence_Fast_GET_ITEM(seq, i)));
    over = __builtin_mul_overflow(*numel, dims->back(), numel) || over;
  }
  if (over) *numel = -1;
  Py_DECREF(seq);
  return !PyErr_Occurred();
}
// Another tensor over the same memory: its shape and strides can be changed in place without changing t's.  Where autograd is not
// involved, without its dispatch (0.1 us in place of 1, and a decode step of 5 us asks for its result once).
at::Tensor alias_of(const at::Tensor& t) {
  if (t.requires_grad() || t.is_inference() || t.unsafeGetTensorImpl()->is_python_dispatch()) return t.alias();
  return at::Tensor(t.unsafeGetTensorImpl()->shallow_copy_and_detach(t.unsafeGetTensorImpl()->version_counter(),
                                                                     /*allow_tensor_metadata_change=*/true));
}
// `t` as the declared precision's values: a tensor of that type itself, or integers of its width, or bytes, that carry its
// bits.  Anything else would be read at a wrong width or as other numbers: undefined, with an exception set.  Of a packed
// buffer longer than `numel` values, its beginning.
at::Tensor as_declared(const at::Tensor& t, PyObject* precision, int64_t numel) {
  if (precision != g_fp32 && precision != g_bf16) {
    PyErr_SetString(PyExc_TypeError, "the precision is Precision.FP32 or Precision.BF16");
    return {};
  }
  const at::ScalarType want = precision == g_bf16 ? at::kBFloat16 : at::kFloat, have = t.scalar_type();
  const bool bits = c10::isIntegralType(have, /*includeBool=*/false) && (t.itemsize() == 1 || t.itemsize() == (want == at::kFloat ? 4 : 2));
  if (!bits && have != want) {
    PyErr_Format(PyExc_TypeError, "a torch tensor of type %s does not hold %s values", c10::toString(have), precision == g_bf16 ? "BF16" : "FP32");
    return {};
  }
  const int64_t per_value = bits ? (want == at::kFloat ? 4 : 2) / t.itemsize() : 1;   // elements of t
  const bool longer = numel >= 0 && t.numel() / per_value >= numel && t.numel() != numel * per_value && t.is_contiguous();
  const at::Tensor part = longer ? t.view(-1).narrow(0, 0, numel * per_value) : t;
  return bits ? part.view(want) : part;
}
PyObject* tensor_set(PyObject* o, PyObject* const* a, Py_ssize_t nargs) {   // torch tensor, logical shape, precision
  if (nargs != 3 || !THPVariable_Check(a[0])) {
    PyErr_SetString(PyExc_TypeError, "a torch tensor, a shape and a precision are needed");
    return nullptr;
  }
  return guard([&]() -> PyObject* {
    c10::SmallVector<int64_t, 6> dims;
    int64_t numel;
    if (!read_shape(a[1], &dims, &numel)) return nullptr;
    const at::Tensor t = as_declared(THPVariable_Unpack(a[0]), a[2], numel);
    if (!t.defined()) return nullptr;
    ten(o) = t.sizes() == at::IntArrayRef(dims) ? alias_of(t) : t.view(dims);
    Py_RETURN_NONE;
  });
}
// An accessor: `f` on the held tensor.  ValueError for an object that holds none (Tensor.__new__ alone); nothing throws past it.
template <typename F>
PyObject* on_held(PyObject* o, F&& f) {
  if (!ten(o).defined()) {
    PyErr_SetString(PyExc_ValueError, "the Tensor holds no storage: its constructor has not run");
    return nullptr;
  }
  return guard([&]() -> PyObject* { return f(ten(o)); });
}
PyObject* tensor_torch(PyObject* o, PyObject*) {
  return on_held(o, [](const at::Tensor& t) { return THPVariable_Wrap(alias_of(t)); });
}
PyObject* tensor_shape(PyObject* o, PyObject*) {
  return on_held(o, [](const at::Tensor& t) {
    const auto s = t.sizes();
    PyObject* r = PyList_New(static_cast<Py_ssize_t>(s.size()));
    for (size_t i = 0; r != nullptr && i < s.size(); ++i) PyList_SET_ITEM(r, i, PyLong_FromLongLong(s[i]));
    return r;
  });
}
PyObject* tensor_precision(PyObject* o, PyObject*) {
  return on_held(o, [](const at::Tensor& t) { return Py_NewRef(is_bf16(t) ? g_bf16 : g_fp32); });
}
PyObject* tensor_numel(PyObject* o, PyObject*) {
  return on_held(o, [](const at::Tensor& t) { return PyLong_FromLongLong(t.numel()); });
}
PyObject* tensor_data_ptr(PyObject* o, PyObject*) {
  return on_held(o, [](const at::Tensor& t) -> PyObject* {
    if (!t.is_contiguous()) {   // the kernels take packed rows, and an address does not tell
      PyErr_SetString(PyExc_ValueError, "the tensor's storage is not contiguous");
      return nullptr;
    }
    return PyLong_FromVoidPtr(t.data_ptr());
  });
}
PyObject* tensor_reshaped(PyObject* o, PyObject* shape) {   // the same memory under another shape; None if the sizes differ
  return on_held(o, [shape](const at::Tensor& t) -> PyObject* {
    c10::SmallVector<int64_t, 6> dims;
    int64_t numel;
    if (!read_shape(shape, &dims, &numel)) return nullptr;
    if (numel != t.numel()) Py_RETURN_NONE;
    return wrap(t.view(dims));
  });
}

PyMethodDef tensor_methods[] = {
    {"_set", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(tensor_set)), METH_FASTCALL, nullptr},
    {"torch", tensor_torch, METH_NOARGS, "The torch tensor behind it, in the logical shape."},
    {"shape", tensor_shape, METH_NOARGS, "The shape, as a list."},
    {"precision", tensor_precision, METH_NOARGS, "Precision.FP32 or Precision.BF16."},
    {"numel", tensor_numel, METH_NOARGS, "Number of elements."},
    {"data_ptr", tensor_data_ptr, METH_NOARGS, "Device address."},
    {"_reshaped", tensor_reshaped, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyMemberDef tensor_members[] = {
    {"lse", T_OBJECT, offsetof(TensorObject, lse), 0, "Side output of the attention ops: per-row log-sum-exp, fp32."},
    {nullptr, 0, 0, 0, nullptr}};
PyTypeObject TensorBaseType = {PyVarObject_HEAD_INIT(nullptr, 0)};

PyObject* setup(PyObject*, PyObject* args) {   // Tensor, Precision.FP32, Precision.BF16, check(status), context(device)
  PyObject *t, *f, *b, *c, *x;
  if (!PyArg_ParseTuple(args, "OOOOO", &t, &f, &b, &c, &x)) return nullptr;
  if (!PyType_Check(t) || !PyType_IsSubtype(reinterpret_cast<PyTypeObject*>(t), g_base)) {
    PyErr_SetString(PyExc_TypeError, "Tensor must derive from TensorBase");
    return nullptr;
  }
  g_tensor = reinterpret_cast<PyTypeObject*>(Py_NewRef(t));
  g_fp32 = Py_NewRef(f);
  g_bf16 = Py_NewRef(b);
  g_check = Py_NewRef(c);
  g_context = Py_NewRef(x);
  Py_RETURN_NONE;
}

#define IT_FN(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {{"setup", setup, METH_VARARGS, nullptr},
                         IT_FN(flash_attention),
                         IT_FN(attention),
                         IT_FN(attention_gqa),
                         IT_FN(attention_backward),
                         IT_FN(attention_backward_recompute),
                         IT_FN(attention_gqa_backward),
                         IT_FN(attention_decode),
                         IT_FN(attention_packed),
                         IT_FN(attention_packed_backward),
                         IT_FN(rope_qk),
                         IT_FN(linear_forward),
                         IT_FN(linear_backward),
                         IT_FN(qkv_rope_forward),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host_ops", "Native host side of the irontensor_b200 ops.", -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__host_ops() {
  TensorBaseType.tp_name = "irontensor_b200._host_ops.TensorBase";
  TensorBaseType.tp_basicsize = sizeof(TensorObject);
  TensorBaseType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_BASETYPE | Py_TPFLAGS_HAVE_GC;
  TensorBaseType.tp_new = tensor_new;
  TensorBaseType.tp_dealloc = [](PyObject* o) {
    if (PyObject_GC_IsTracked(o)) PyObject_GC_UnTrack(o);
    tensor_dealloc(o);
  };
  TensorBaseType.tp_traverse = tensor_traverse;
  TensorBaseType.tp_clear = tensor_clear;
  TensorBaseType.tp_methods = tensor_methods;
  TensorBaseType.tp_members = tensor_members;
  if (PyType_Ready(&TensorBaseType) < 0) return nullptr;
  g_base = &TensorBaseType;
  PyObject* m = PyModule_Create(&module);
  if (m != nullptr && PyModule_AddObjectRef(m, "TensorBase", reinterpret_cast<PyObject*>(g_base)) < 0) Py_CLEAR(m);
  return m;
}
