// The host side of a layer call as one native function per entry point.
//
// A decode-sized call is 3-9 us of GPU work.  Walked in Python -- argument checks, torch.empty,
// data_ptr(), a ctypes call with a dozen converted arguments, a device context -- its host side took
// 15 us (and 12-20 us more for every quantizer or GEMM entry point called by itself), so the GPU
// waited for the host at every size below a few hundred tokens.  Here the checks, the output
// allocation, the workspace lookup and the library call are one METH_FASTCALL function.
//
// Every function handles the plain case -- bf16 CUDA tensors of the layer's device with unit inner
// stride, shapes that match -- and returns None otherwise without having launched anything; the
// caller (linear.py, activation.py) then takes the general route, which converts what can be
// converted and raises the errors.  The calls only enqueue work and keep the GIL, which keeps the two
// launches of a forward together when two threads share a stream.  forward_host releases it: a copy from
// or to pageable memory waits for the stream, and a lock per scratch set keeps its launches together.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <map>
#include <mutex>
#include <optional>
#include <unordered_map>
#include <utility>

#include "internal.h"

namespace {

// ---------------------------------------------------------------- scratch per (device, stream)
// Calls on one stream are ordered and share a set; calls on different streams may overlap on the
// GPU, so each stream has its own.  Grown on demand, at most one set per stream of the process
// (PyTorch hands out a fixed pool of streams).  Never destroyed at exit: the tensors must not
// outlive the CUDA context's teardown order.
struct Workspace {
  at::Tensor ws;            // zero-initialised: arrival counters lead, then kernel scratch
  at::Tensor q, scale;      // quantized activations of a forward
  at::Tensor host_scratch;  // everything a host-buffer forward needs on the device
  std::mutex host_lock;     // ... and whose turn it is to use it; taken without the GIL only
};

std::map<std::pair<int, cudaStream_t>, Workspace>& pool() {
  static auto* p = new std::map<std::pair<int, cudaStream_t>, Workspace>();
  return *p;
}

at::Tensor new_tensor(at::IntArrayRef size, at::ScalarType t, int dev) {
  return at::Tensor(at::detail::empty_cuda(size, t, c10::Device(c10::kCUDA, (c10::DeviceIndex)dev), std::nullopt));
}

at::Tensor zeroed(int64_t bytes, int dev) { return new_tensor({bytes}, at::kByte, dev).zero_(); }

Workspace& workspace(int dev, cudaStream_t s) {
  static thread_local std::pair<int, cudaStream_t> last_key{-1, nullptr};
  static thread_local Workspace* last = nullptr;
  const std::pair<int, cudaStream_t> key{dev, s};
  if (last == nullptr || key != last_key) {
    last = &pool()[key];                              // map nodes do not move
    last_key = key;
  }
  return *last;
}

at::Tensor& scratch(Workspace& w, int64_t bytes, int dev) {
  if (!w.ws.defined() || w.ws.numel() < bytes) w.ws = zeroed(bytes > (1 << 20) ? bytes : (1 << 20), dev);
  return w.ws;
}

void act_buffers(Workspace& w, int64_t m, int64_t k, int dev) {
  if (!w.q.defined() || w.q.numel() < m * k) w.q = new_tensor({m * k > (1 << 16) ? m * k : (1 << 16)}, at::kByte, dev);
  if (!w.scale.defined() || w.scale.numel() < m) w.scale = new_tensor({m > 1024 ? m : 1024}, at::kFloat, dev);
}

// ---------------------------------------------------------------- small helpers
PyObject* g_error_class = nullptr;   // sacq_b200._lib.SacqError(code, message)

PyObject* raise_status(int rc) {
  PyObject* args = Py_BuildValue("(is)", rc, sacq_last_error());
  if (args != nullptr) {
    PyObject* e = PyObject_CallObject(g_error_class ? g_error_class : PyExc_RuntimeError, args);
    Py_DECREF(args);
    if (e != nullptr) {
      PyErr_SetObject((PyObject*)Py_TYPE(e), e);
      Py_DECREF(e);
    }
  }
  return nullptr;
}

const at::Tensor* tensor_of(PyObject* o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }

bool on_device(const at::Tensor& t, int dev) { return t.is_cuda() && t.get_device() == dev; }

// A 2-D tensor whose rows are contiguous (the inner stride of rows of one element means nothing).
bool whole_rows(const at::Tensor& t) { return t.dim() == 2 && (t.stride(1) == 1 || t.size(1) == 1); }

// bf16 [m, k] rows with unit inner stride
bool bf16_rows(const at::Tensor& t, int dev) {
  return t.scalar_type() == at::kBFloat16 && on_device(t, dev) && whole_rows(t);
}

bool f32_vector(const at::Tensor& t, int64_t n, int dev) {
  return t.scalar_type() == at::kFloat && on_device(t, dev) && t.numel() == n && t.is_contiguous();
}

bool byte_matrix(const at::Tensor& t, int64_t k, int dev) {
  return t.element_size() == 1 && on_device(t, dev) && t.dim() == 2 && t.size(1) == k && t.is_contiguous();
}

// The stream work of a device goes to, and that device made current while the object lives.
struct Target {
  int dev;
  cudaStream_t stream;
  std::optional<c10::cuda::CUDAGuard> guard;
  explicit Target(int d) : dev(d), stream(c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)d).stream()) {
    if (c10::cuda::current_device() != d) guard.emplace((c10::DeviceIndex)d);
  }
};

// A C++ exception leaves as the Python exception that PyTorch makes of it (an allocation that fails as
// torch.OutOfMemoryError, which callers catch to free memory and try again).
#define NATIVE_TRY try {
#define NATIVE_CATCH                                                                            \
  }                                                                                             \
  catch (...) {                                                                                 \
    if (!PyErr_Occurred()) torch::translate_exception_to_python(std::current_exception());      \
    return nullptr;                                                                             \
  }

// Activations of a forward: any [..., K] bf16 tensor whose rows can be addressed with one pitch.
struct Rows {
  const void* ptr;
  int64_t m, pitch;
};

bool rows_of(const at::Tensor& x, int64_t k, int dev, Rows& r) {
  const int64_t nd = x.dim();
  if (nd < 1 || x.scalar_type() != at::kBFloat16 || !on_device(x, dev) || x.size(nd - 1) != k) return false;
  if (nd == 2) {
    if (!whole_rows(x)) return false;
    r = {x.data_ptr(), x.size(0), x.stride(0)};
  } else {
    if (!x.is_contiguous()) return false;
    r = {x.data_ptr(), k > 0 ? x.numel() / k : 0, k};
  }
  return r.m > 0;
}

// [..., n] like x, for a fresh [m, n] result
at::Tensor result_like(const at::Tensor& x, int64_t m, int64_t n, int dev) {
  if (x.dim() == 2) return new_tensor({m, n}, at::kBFloat16, dev);
  c10::SmallVector<int64_t, 8> shape(x.sizes().begin(), x.sizes().end());
  shape.back() = n;
  return new_tensor(shape, at::kBFloat16, dev);
}

// ---------------------------------------------------------------- one layer
enum NeedKind { kNeedA8 = 0, kNeedInt8 = 1, kNeedHost = 2, kNeedKinds = 3 };

struct LayerObject {
  PyObject_HEAD
  sacq_layer_t* handle;      // borrowed from the Python module that owns both
  int dev;
  int64_t k, n;
  std::unordered_map<int64_t, int64_t>* need;   // workspace bytes by 3 * M + kind
};

int64_t need_bytes(LayerObject* L, int64_t m, NeedKind kind) {
  const int64_t key = m * kNeedKinds + kind;
  auto it = L->need->find(key);
  if (it != L->need->end()) return it->second;
  const int64_t b = kind == kNeedA8     ? sacq_workspace_bytes(L->handle, m)
                    : kind == kNeedInt8 ? sacq_workspace_bytes_int8(L->handle, m)
                                        : sacq_host_forward_scratch_bytes(L->handle, m);
  if (L->need->size() > 4096) L->need->clear();       // a program with ragged token counts does not grow it without end
  L->need->emplace(key, b);
  return b;
}

// out (None, or a bf16 [m, n] tensor with unit inner stride on the device) -> the tensor to write, or undefined
at::Tensor out_or_new(PyObject* out, int64_t m, int64_t n, int dev) {
  if (out == Py_None) return new_tensor({m, n}, at::kBFloat16, dev);
  const at::Tensor* t = tensor_of(out);
  if (t == nullptr || !bf16_rows(*t, dev) || t->size(0) != m || t->size(1) != n) return at::Tensor();
  return *t;
}

PyObject* layer_forward(LayerObject* L, PyObject* x_obj) {
  NATIVE_TRY
  const at::Tensor* x = tensor_of(x_obj);
  Rows r;
  if (x == nullptr || L->n <= 0 || !rows_of(*x, L->k, L->dev, r)) Py_RETURN_NONE;
  Target at_(L->dev);
  Workspace& w = workspace(L->dev, at_.stream);
  at::Tensor& ws = scratch(w, need_bytes(L, r.m, kNeedA8), L->dev);
  act_buffers(w, r.m, L->k, L->dev);
  at::Tensor y = result_like(*x, r.m, L->n, L->dev);
  const int rc = sacq_forward_call(L->handle, r.ptr, r.pitch, r.m, 0, nullptr, 0, w.q.data_ptr(), (float*)w.scale.data_ptr(),
                                   y.data_ptr(), L->n, ws.data_ptr(), ws.numel(), at_.stream);
  return rc == 0 ? THPVariable_Wrap(std::move(y)) : raise_status(rc);
  NATIVE_CATCH
}

PyObject* layer_forward_residual(LayerObject* L, PyObject* const* a, Py_ssize_t n) {
  NATIVE_TRY
  const at::Tensor *x = n == 2 ? tensor_of(a[0]) : nullptr, *res = n == 2 ? tensor_of(a[1]) : nullptr;
  Rows r, rr;
  if (x == nullptr || res == nullptr || L->n <= 0 || !rows_of(*x, L->k, L->dev, r) || !rows_of(*res, L->n, L->dev, rr) ||
      rr.m != r.m)
    Py_RETURN_NONE;
  Target at_(L->dev);
  Workspace& w = workspace(L->dev, at_.stream);
  at::Tensor& ws = scratch(w, need_bytes(L, r.m, kNeedA8), L->dev);
  act_buffers(w, r.m, L->k, L->dev);
  at::Tensor y = result_like(*x, r.m, L->n, L->dev);
  const int rc = sacq_forward_call(L->handle, r.ptr, r.pitch, r.m, 0, rr.ptr, rr.pitch, w.q.data_ptr(),
                                   (float*)w.scale.data_ptr(), y.data_ptr(), L->n, ws.data_ptr(), ws.numel(), at_.stream);
  return rc == 0 ? THPVariable_Wrap(std::move(y)) : raise_status(rc);
  NATIVE_CATCH
}

PyObject* layer_forward_int8(LayerObject* L, PyObject* x_obj) {
  NATIVE_TRY
  const at::Tensor* x = tensor_of(x_obj);
  Rows r;
  if (x == nullptr || L->n <= 0 || !rows_of(*x, L->k, L->dev, r)) Py_RETURN_NONE;
  Target at_(L->dev);
  Workspace& w = workspace(L->dev, at_.stream);
  at::Tensor& ws = scratch(w, need_bytes(L, r.m, kNeedInt8), L->dev);
  act_buffers(w, r.m, L->k, L->dev);
  at::Tensor y = result_like(*x, r.m, L->n, L->dev);
  const int rc = sacq_forward_call(L->handle, r.ptr, r.pitch, r.m, 1, nullptr, 0, w.q.data_ptr(), (float*)w.scale.data_ptr(),
                                   y.data_ptr(), L->n, ws.data_ptr(), ws.numel(), at_.stream);
  return rc == 0 ? THPVariable_Wrap(std::move(y)) : raise_status(rc);
  NATIVE_CATCH
}

// linear_a8(q, scale, out, residual, int8)
PyObject* layer_linear_a8(LayerObject* L, PyObject* const* a, Py_ssize_t n) {
  NATIVE_TRY
  const at::Tensor *q = n == 5 ? tensor_of(a[0]) : nullptr, *s = n == 5 ? tensor_of(a[1]) : nullptr;
  if (q == nullptr || s == nullptr || L->n <= 0 || !byte_matrix(*q, L->k, L->dev)) Py_RETURN_NONE;
  const int64_t m = q->size(0);
  const bool int8 = a[4] == Py_True;
  if (m == 0 || !f32_vector(*s, m, L->dev) || (int8 && q->scalar_type() != at::kChar)) Py_RETURN_NONE;
  const at::Tensor* res = nullptr;
  if (a[3] != Py_None) {
    res = tensor_of(a[3]);
    if (res == nullptr || int8 || !bf16_rows(*res, L->dev) || res->size(0) != m || res->size(1) != L->n) Py_RETURN_NONE;
  }
  Target at_(L->dev);
  at::Tensor y = out_or_new(a[2], m, L->n, L->dev);
  if (!y.defined()) Py_RETURN_NONE;
  at::Tensor& ws = scratch(workspace(L->dev, at_.stream), need_bytes(L, m, int8 ? kNeedInt8 : kNeedA8), L->dev);
  const void* qp = q->data_ptr();
  const float* sp = (const float*)s->data_ptr();
  const int rc =
      int8 ? sacq_linear_a8i(L->handle, qp, sp, m, y.data_ptr(), y.stride(0), ws.data_ptr(), ws.numel(), at_.stream)
      : res ? sacq_linear_a8_residual(L->handle, qp, sp, m, res->data_ptr(), res->stride(0), y.data_ptr(), y.stride(0),
                                      ws.data_ptr(), ws.numel(), at_.stream)
            : sacq_linear_a8(L->handle, qp, sp, m, y.data_ptr(), y.stride(0), ws.data_ptr(), ws.numel(), at_.stream);
  return rc == 0 ? THPVariable_Wrap(std::move(y)) : raise_status(rc);
  NATIVE_CATCH
}

// linear_w8a8(q, scale, weight_row_scale, out, int8)
PyObject* layer_linear_w8a8(LayerObject* L, PyObject* const* a, Py_ssize_t n) {
  NATIVE_TRY
  const at::Tensor *q = n == 5 ? tensor_of(a[0]) : nullptr, *s = n == 5 ? tensor_of(a[1]) : nullptr,
                   *sw = n == 5 ? tensor_of(a[2]) : nullptr;
  if (q == nullptr || s == nullptr || sw == nullptr || L->n <= 0 || !byte_matrix(*q, L->k, L->dev)) Py_RETURN_NONE;
  const int64_t m = q->size(0);
  const bool int8 = a[4] == Py_True;
  const at::ScalarType t = q->scalar_type();
  if (m == 0 || !f32_vector(*s, m, L->dev) || !f32_vector(*sw, L->n, L->dev) ||
      !(int8 ? t == at::kChar : (t == at::kFloat8_e4m3fn || t == at::kByte)))
    Py_RETURN_NONE;
  Target at_(L->dev);
  at::Tensor y = out_or_new(a[3], m, L->n, L->dev);
  if (!y.defined()) Py_RETURN_NONE;
  at::Tensor& ws = scratch(workspace(L->dev, at_.stream), sacq_workspace_bytes_w8a8(L->handle, m), L->dev);
  const int rc = (int8 ? sacq_linear_w8a8_int8 : sacq_linear_w8a8_fp8)(
      L->handle, q->data_ptr(), (const float*)s->data_ptr(), (const float*)sw->data_ptr(), m, y.data_ptr(), y.stride(0),
      ws.data_ptr(), ws.numel(), at_.stream);
  return rc == 0 ? THPVariable_Wrap(std::move(y)) : raise_status(rc);
  NATIVE_CATCH
}

// forward_host(x_host, out_host): both CPU bf16, contiguous
PyObject* layer_forward_host(LayerObject* L, PyObject* const* a, Py_ssize_t n) {
  NATIVE_TRY
  const at::Tensor *x = n == 2 ? tensor_of(a[0]) : nullptr, *y = n == 2 ? tensor_of(a[1]) : nullptr;
  if (x == nullptr || y == nullptr || L->n <= 0 || !x->is_cpu() || !y->is_cpu() || x->scalar_type() != at::kBFloat16 ||
      y->scalar_type() != at::kBFloat16 || x->dim() != 2 || y->dim() != 2 || !x->is_contiguous() || !y->is_contiguous() ||
      x->size(1) != L->k || x->size(0) <= 0 || y->size(0) != x->size(0) || y->size(1) != L->n)
    Py_RETURN_NONE;
  const int64_t m = x->size(0);
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)L->dev).stream();
  Workspace& w = workspace(L->dev, stream);
  const int64_t need = need_bytes(L, m, kNeedHost);
  if (!w.host_scratch.defined() || w.host_scratch.numel() < need) {
    Target at_(L->dev);
    w.host_scratch = zeroed(need > (1 << 22) ? need : (1 << 22), L->dev);
  }
  // the call's own references: another thread may let go of its tensors, or grow the scratch, meanwhile
  const at::Tensor xt = *x, yt = *y, scratch_t = w.host_scratch;
  const void* xp = xt.data_ptr();
  void *yp = yt.data_ptr(), *sp = scratch_t.data_ptr();
  const int64_t bytes = scratch_t.numel();
  int rc;
  Py_BEGIN_ALLOW_THREADS
  {
    std::lock_guard<std::mutex> turn(w.host_lock);
    // the library switches to the layer's device itself
    rc = sacq_linear_bf16_host(L->handle, xp, m, yp, sp, bytes, stream);
  }
  Py_END_ALLOW_THREADS
  if (rc != 0) return raise_status(rc);
  Py_INCREF(a[1]);
  return a[1];
  NATIVE_CATCH
}

PyObject* layer_forget(LayerObject* L, PyObject*) {   // the kernel choice changed: so may the workspace sizes
  L->need->clear();
  Py_RETURN_NONE;
}

PyMethodDef layer_methods[] = {
    {"forward", (PyCFunction)layer_forward, METH_O, nullptr},
    {"forward_residual", (PyCFunction)(void*)layer_forward_residual, METH_FASTCALL, nullptr},
    {"forward_int8", (PyCFunction)layer_forward_int8, METH_O, nullptr},
    {"linear_a8", (PyCFunction)(void*)layer_linear_a8, METH_FASTCALL, nullptr},
    {"linear_w8a8", (PyCFunction)(void*)layer_linear_w8a8, METH_FASTCALL, nullptr},
    {"forward_host", (PyCFunction)(void*)layer_forward_host, METH_FASTCALL, nullptr},
    {"forget_sizes", (PyCFunction)layer_forget, METH_NOARGS, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyObject* layer_new(PyTypeObject* type, PyObject* args, PyObject*) {
  unsigned long long handle = 0;
  int dev = 0;
  long long n = 0, k = 0;
  if (!PyArg_ParseTuple(args, "KiLL", &handle, &dev, &n, &k)) return nullptr;
  LayerObject* L = (LayerObject*)type->tp_alloc(type, 0);
  if (L == nullptr) return nullptr;
  L->handle = (sacq_layer_t*)(uintptr_t)handle;
  L->dev = dev;
  L->n = n;
  L->k = k;
  L->need = new std::unordered_map<int64_t, int64_t>();
  return (PyObject*)L;
}

void layer_dealloc(LayerObject* L) {
  delete L->need;
  Py_TYPE(L)->tp_free((PyObject*)L);
}

PyTypeObject LayerType = {PyVarObject_HEAD_INIT(nullptr, 0)};

// ---------------------------------------------------------------- quantizers
PyObject* pair_of(at::Tensor q, at::Tensor s) {
  PyObject* t = PyTuple_New(2);
  PyObject *a = THPVariable_Wrap(std::move(q)), *b = THPVariable_Wrap(std::move(s));
  if (t == nullptr || a == nullptr || b == nullptr) {
    Py_XDECREF(t);
    Py_XDECREF(a);
    Py_XDECREF(b);
    return nullptr;
  }
  PyTuple_SET_ITEM(t, 0, a);
  PyTuple_SET_ITEM(t, 1, b);
  return t;
}

// Fresh (q [m, k], scale [m, 1])
struct Encoded {
  at::Tensor q, s;
  Encoded(int64_t m, int64_t k, bool int8, int dev)
      : q(new_tensor({m, k}, int8 ? at::kChar : at::kFloat8_e4m3fn, dev)), s(new_tensor({m, 1}, at::kFloat, dev)) {}
};

// The 2-D bf16 CUDA input of a quantizer, not empty
const at::Tensor* quantizer_input(PyObject* o) {
  const at::Tensor* x = tensor_of(o);
  if (x == nullptr || !x->is_cuda() || !bf16_rows(*x, x->get_device()) || x->numel() == 0) return nullptr;
  return x;
}

// A bf16 vector of k contiguous elements, null for None; false: not that
bool vector_or_none(PyObject* o, int64_t k, int dev, const void** p) {
  *p = nullptr;
  if (o == Py_None) return true;
  const at::Tensor* t = tensor_of(o);
  if (t == nullptr || t->scalar_type() != at::kBFloat16 || !on_device(*t, dev) || t->numel() != k || !t->is_contiguous())
    return false;
  *p = t->data_ptr();
  return true;
}

// quantize_rows(x, int8)
PyObject* py_quantize_rows(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_TRY
  const at::Tensor* x = n == 2 ? quantizer_input(a[0]) : nullptr;
  if (x == nullptr) Py_RETURN_NONE;
  const bool int8 = a[1] == Py_True;
  Target at_(x->get_device());
  Encoded e(x->size(0), x->size(1), int8, at_.dev);
  const int rc = (int8 ? sacq_quant_act_int8 : sacq_quant_act_fp8)(x->data_ptr(), x->stride(0), x->size(0), x->size(1),
                                                                   e.q.data_ptr(), (float*)e.s.data_ptr(), at_.stream);
  return rc == 0 ? pair_of(std::move(e.q), std::move(e.s)) : raise_status(rc);
  NATIVE_CATCH
}

// act_quantize_rows(kind, a, b)
PyObject* py_act_quantize_rows(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_TRY
  const at::Tensor* x = n == 3 ? quantizer_input(a[1]) : nullptr;
  if (x == nullptr) Py_RETURN_NONE;
  const long kind = PyLong_AsLong(a[0]);
  const at::Tensor* b = nullptr;
  if (kind == SACQ_ACT_SILU_MUL) {
    b = tensor_of(a[2]);
    if (b == nullptr || !bf16_rows(*b, x->get_device()) || b->sizes() != x->sizes()) Py_RETURN_NONE;
  }
  Target at_(x->get_device());
  Encoded e(x->size(0), x->size(1), false, at_.dev);
  const int rc = sacq_act_quant_fp8((int)kind, x->data_ptr(), x->stride(0), b ? b->data_ptr() : nullptr,
                                    b ? b->stride(0) : 0, x->size(0), x->size(1), e.q.data_ptr(), (float*)e.s.data_ptr(),
                                    at_.stream);
  return rc == 0 ? pair_of(std::move(e.q), std::move(e.s)) : raise_status(rc);
  NATIVE_CATCH
}

// modulate_quantize_rows(x, scale, shift)
PyObject* py_modulate_quantize_rows(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_TRY
  const at::Tensor* x = n == 3 ? quantizer_input(a[0]) : nullptr;
  const void *sc = nullptr, *sh = nullptr;
  if (x == nullptr || !vector_or_none(a[1], x->size(1), x->get_device(), &sc) ||
      !vector_or_none(a[2], x->size(1), x->get_device(), &sh) || sc == nullptr || sh == nullptr)
    Py_RETURN_NONE;
  Target at_(x->get_device());
  Encoded e(x->size(0), x->size(1), false, at_.dev);
  const int rc = sacq_modulate_quant_fp8(x->data_ptr(), x->stride(0), sc, sh, x->size(0), x->size(1), e.q.data_ptr(),
                                         (float*)e.s.data_ptr(), at_.stream);
  return rc == 0 ? pair_of(std::move(e.q), std::move(e.s)) : raise_status(rc);
  NATIVE_CATCH
}

// layernorm_quantize_rows(x, weight, bias, eps, mod_scale, mod_shift, return_normalized)
PyObject* py_layernorm_quantize_rows(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_TRY
  const at::Tensor* x = n == 7 ? quantizer_input(a[0]) : nullptr;
  if (x == nullptr) Py_RETURN_NONE;
  const int64_t m = x->size(0), k = x->size(1);
  const int dev = x->get_device();
  const void* v[4];
  static const int at_arg[4] = {1, 2, 4, 5};
  for (int i = 0; i < 4; ++i)
    if (!vector_or_none(a[at_arg[i]], k, dev, &v[i])) Py_RETURN_NONE;
  if ((v[2] == nullptr) != (v[3] == nullptr)) Py_RETURN_NONE;
  const double eps = PyFloat_AsDouble(a[3]);
  if (eps == -1.0 && PyErr_Occurred()) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  const int want_y = PyObject_IsTrue(a[6]);            // any truth value, as the general route takes it
  if (want_y < 0) return nullptr;
  Target at_(dev);
  Encoded e(m, k, false, dev);
  at::Tensor y;
  if (want_y) y = new_tensor({m, k}, at::kBFloat16, dev);
  const int rc = sacq_layernorm_quant_fp8(x->data_ptr(), x->stride(0), v[0], v[1], (float)eps, v[2], v[3], m, k,
                                          y.defined() ? y.data_ptr() : nullptr, k, e.q.data_ptr(), (float*)e.s.data_ptr(),
                                          at_.stream);
  if (rc != 0) return raise_status(rc);
  if (!y.defined()) return pair_of(std::move(e.q), std::move(e.s));
  PyObject *q = THPVariable_Wrap(std::move(e.q)), *s = THPVariable_Wrap(std::move(e.s)), *yy = THPVariable_Wrap(std::move(y));
  PyObject* t = (q && s && yy) ? PyTuple_Pack(3, q, s, yy) : nullptr;
  Py_XDECREF(q);
  Py_XDECREF(s);
  Py_XDECREF(yy);
  return t;
  NATIVE_CATCH
}

// ---------------------------------------------------------------- several layers on one input
constexpr int kMostSiblings = 16;

struct Siblings {
  LayerObject* L[kMostSiblings];
  int n = 0;
};

// A list of modules that carry a Layer as `_native`, all of one device and input width
bool siblings_of(PyObject* list, Siblings& out) {
  static PyObject* name = PyUnicode_InternFromString("_native");
  if (!PyList_Check(list)) return false;
  const Py_ssize_t n = PyList_GET_SIZE(list);
  if (n < 1 || n > kMostSiblings) return false;
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* o = PyObject_GetAttr(PyList_GET_ITEM(list, i), name);
    if (o == nullptr) {
      PyErr_Clear();
      return false;
    }
    const bool ok = Py_TYPE(o) == &LayerType;
    Py_DECREF(o);                                     // the module keeps it
    if (!ok) return false;
    out.L[i] = (LayerObject*)o;
    if (out.L[i]->k != out.L[0]->k || out.L[i]->dev != out.L[0]->dev || out.L[i]->n <= 0) return false;
  }
  out.n = (int)n;
  return true;
}

PyObject* run_siblings(const Siblings& sb, const void* q, const float* s, int64_t m, const at::Tensor* like,
                       const Target& at_) {
  int64_t need = 0;
  const sacq_layer_t* handles[kMostSiblings];
  void* ys[kMostSiblings];
  int64_t ldys[kMostSiblings];
  at::Tensor outs[kMostSiblings];
  for (int i = 0; i < sb.n; ++i) {
    LayerObject* L = sb.L[i];
    need = std::max(need, need_bytes(L, m, kNeedA8));
    handles[i] = L->handle;
    outs[i] = like ? result_like(*like, m, L->n, L->dev) : new_tensor({m, L->n}, at::kBFloat16, L->dev);
    ys[i] = outs[i].data_ptr();
    ldys[i] = L->n;
  }
  at::Tensor& ws = scratch(workspace(at_.dev, at_.stream), need, at_.dev);
  const int rc = sacq_linear_a8_multi(handles, sb.n, q, s, m, ys, ldys, ws.data_ptr(), ws.numel(), at_.stream);
  if (rc != 0) return raise_status(rc);
  PyObject* list = PyList_New(sb.n);
  for (int i = 0; i < sb.n && list != nullptr; ++i) {
    PyObject* o = THPVariable_Wrap(std::move(outs[i]));
    if (o == nullptr) {
      Py_DECREF(list);
      return nullptr;
    }
    PyList_SET_ITEM(list, i, o);
  }
  return list;
}

// linear_a8_multi(layers, q, scale)
PyObject* py_linear_a8_multi(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_TRY
  Siblings sb;
  const at::Tensor *q = n == 3 ? tensor_of(a[1]) : nullptr, *s = n == 3 ? tensor_of(a[2]) : nullptr;
  if (q == nullptr || s == nullptr || !siblings_of(a[0], sb) || !byte_matrix(*q, sb.L[0]->k, sb.L[0]->dev) ||
      q->size(0) == 0 || !f32_vector(*s, q->size(0), sb.L[0]->dev))
    Py_RETURN_NONE;
  Target at_(sb.L[0]->dev);
  return run_siblings(sb, q->data_ptr(), (const float*)s->data_ptr(), q->size(0), nullptr, at_);
  NATIVE_CATCH
}

// forward_shared(layers, x)
PyObject* py_forward_shared(PyObject*, PyObject* const* a, Py_ssize_t n) {
  NATIVE_TRY
  Siblings sb;
  Rows r;
  const at::Tensor* x = n == 2 ? tensor_of(a[1]) : nullptr;
  if (x == nullptr || !siblings_of(a[0], sb) || !rows_of(*x, sb.L[0]->k, sb.L[0]->dev, r)) Py_RETURN_NONE;
  Target at_(sb.L[0]->dev);
  Workspace& w = workspace(at_.dev, at_.stream);
  act_buffers(w, r.m, sb.L[0]->k, at_.dev);
  const int rc = sacq_quant_act_fp8(r.ptr, r.pitch, r.m, sb.L[0]->k, w.q.data_ptr(), (float*)w.scale.data_ptr(), at_.stream);
  if (rc != 0) return raise_status(rc);
  return run_siblings(sb, w.q.data_ptr(), (const float*)w.scale.data_ptr(), r.m, x, at_);
  NATIVE_CATCH
}

// ---------------------------------------------------------------- the pool, for the general route
// workspace(device, bytes): the current stream's kernel scratch, grown to `bytes`
PyObject* py_workspace(PyObject*, PyObject* args) {
  NATIVE_TRY
  int dev = 0;
  long long bytes = 0;
  if (!PyArg_ParseTuple(args, "iL", &dev, &bytes)) return nullptr;
  Target at_(dev);
  return THPVariable_Wrap(scratch(workspace(dev, at_.stream), bytes, dev));
  NATIVE_CATCH
}

// host_scratch(device, bytes): device scratch of the current stream's host-buffer forwards
PyObject* py_host_scratch(PyObject*, PyObject* args) {
  NATIVE_TRY
  int dev = 0;
  long long bytes = 0;
  if (!PyArg_ParseTuple(args, "iL", &dev, &bytes)) return nullptr;
  Target at_(dev);
  Workspace& w = workspace(dev, at_.stream);
  if (!w.host_scratch.defined() || w.host_scratch.numel() < bytes)
    w.host_scratch = zeroed(bytes > (1 << 22) ? bytes : (1 << 22), dev);
  return THPVariable_Wrap(w.host_scratch);
  NATIVE_CATCH
}

PyObject* py_set_error_class(PyObject*, PyObject* cls) {
  Py_INCREF(cls);
  Py_XSETREF(g_error_class, cls);
  Py_RETURN_NONE;
}

PyMethodDef module_methods[] = {
    {"quantize_rows", (PyCFunction)(void*)py_quantize_rows, METH_FASTCALL, nullptr},
    {"act_quantize_rows", (PyCFunction)(void*)py_act_quantize_rows, METH_FASTCALL, nullptr},
    {"modulate_quantize_rows", (PyCFunction)(void*)py_modulate_quantize_rows, METH_FASTCALL, nullptr},
    {"layernorm_quantize_rows", (PyCFunction)(void*)py_layernorm_quantize_rows, METH_FASTCALL, nullptr},
    {"linear_a8_multi", (PyCFunction)(void*)py_linear_a8_multi, METH_FASTCALL, nullptr},
    {"forward_shared", (PyCFunction)(void*)py_forward_shared, METH_FASTCALL, nullptr},
    {"workspace", py_workspace, METH_VARARGS, nullptr},
    {"host_scratch", py_host_scratch, METH_VARARGS, nullptr},
    {"set_error_class", py_set_error_class, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, module_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) {
  LayerType.tp_name = "sacq_b200._native.Layer";
  LayerType.tp_basicsize = sizeof(LayerObject);
  LayerType.tp_flags = Py_TPFLAGS_DEFAULT;
  LayerType.tp_new = layer_new;
  LayerType.tp_dealloc = (destructor)layer_dealloc;
  LayerType.tp_methods = layer_methods;
  if (PyType_Ready(&LayerType) < 0) return nullptr;
  PyObject* m = PyModule_Create(&module_def);
  if (m == nullptr) return nullptr;
  Py_INCREF(&LayerType);
  if (PyModule_AddObject(m, "Layer", (PyObject*)&LayerType) < 0) {
    Py_DECREF(&LayerType);
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
