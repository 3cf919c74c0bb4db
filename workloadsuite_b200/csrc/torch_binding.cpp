// The short way from PyTorch tensors to the C ABI of ssd_b200.h.  A call of a few microseconds on the GPU (one decoded
// token, a small layer) is otherwise bound by what Python spends on attribute look-ups, ctypes marshalling and context
// managers: 15-20 us per call, against 2-3 us here.
// Every function returns None when the call is not plainly valid for the kernels (other dtypes, shapes that disagree,
// tensors that have to be copied first, a code that says so); the Python wrapper then goes its long way, which copies what
// has to be copied or raises.  Nothing is decided here that the long way would decide otherwise.  A CUDA error is raised
// here: work may have been enqueued by then, and a step made again would advance the state twice.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "ssd_b200.h"

namespace {

using at::Tensor;

// The entry points stand between HANDLE_TH_ERRORS and END_HANDLE_TH_ERRORS from their first line on: what PyTorch's C++ throws
// (a nested tensor has no sizes, an allocation runs out of memory) becomes the Python exception that PyTorch itself raises
// for it, and would end the process if it left the entry point.

// entry points of the library that the Python side has loaded
decltype(&ssd_b200_forward) f_forward;
decltype(&ssd_b200_workspace_bytes) f_workspace;
decltype(&ssd_b200_step_strided) f_step;
decltype(&ssd_b200_conv1d_silu) f_conv;
decltype(&ssd_b200_dt_prologue) f_dt;
PyObject* f_raise;   // raises the Python exception of an error code

constexpr int kMaxDevices = 64;
Tensor* g_workspace[kMaxDevices];   // scratch of the runs that leave results for a later one (never shrinks)
Tensor* g_status[kMaxDevices];      // the kernels' status word

int dtype_of(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return SSD_DTYPE_F32;
    case at::kHalf: return SSD_DTYPE_F16;
    case at::kBFloat16: return SSD_DTYPE_BF16;
    default: return -1;
  }
}

// The tensor behind a Python object: false for anything but a plain tensor; None gives an undefined tensor.
bool get(PyObject* o, const Tensor** out, bool optional = false) {
  static const Tensor none;
  if (o == Py_None) {
    *out = &none;
    return optional;
  }
  if (!THPVariable_CheckExact(o)) return false;
  *out = &THPVariable_Unpack(o);
  return true;
}

bool shaped(const Tensor& t, std::initializer_list<int64_t> s) { return t.sizes() == at::IntArrayRef(s.begin(), s.size()); }
bool inner(const Tensor& t) { return t.stride(-1) == 1 || t.size(-1) == 1; }

// The result of a call that returned `rc`: None, for the long way, unless that could enqueue work twice.
PyObject* declined(int rc) {
  if (rc != SSD_ERR_CUDA) Py_RETURN_NONE;
  Py_XDECREF(PyObject_CallFunction(f_raise, "i", rc));
  return nullptr;
}

struct Where {
  c10::cuda::OptionalCUDAGuard guard;
  c10::Device dev;
  explicit Where(const Tensor& t) : dev(t.device()) { if (c10::cuda::current_device() != dev.index()) guard.set_device(dev); }
  bool here(const Tensor& t) const { return !t.defined() || t.device() == dev; }
  void* stream() const { return c10::cuda::getCurrentCUDAStream(dev.index()).stream(); }
};

Tensor& status_word(int dev) {
  if (!g_status[dev]) g_status[dev] = new Tensor(at::zeros({1024}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, dev)));
  return *g_status[dev];
}
Tensor& workspace(int dev, int64_t bytes) {
  if (!g_workspace[dev] || g_workspace[dev]->numel() < bytes) {
    delete g_workspace[dev];
    g_workspace[dev] = nullptr;
    g_workspace[dev] = new Tensor(at::empty({bytes}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA, dev)));
  }
  return *g_workspace[dev];
}

// Strides of the three outer axes; a size-1 axis gets its contiguous stride (its own is arbitrary and may break the
// 16-byte rule of TMA descriptors).
void strides4(const Tensor& t, int64_t* st) {
  int64_t in = t.size(3);
  for (int d = 2; d >= 0; --d) {
    st[d] = t.size(d) == 1 ? in : t.stride(d);
    in = std::max(in, st[d] * t.size(d));
  }
}
void strides3(const Tensor& t, int64_t* st) {
  for (int d = 0; d < 3; ++d) st[d] = t.stride(d);
}

// step(x, a, B, C, state, dt, D, z, out) -> y
PyObject* py_step(PyObject*, PyObject* const* o, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Tensor *x, *a, *B, *C, *state, *dt, *D, *z, *out;
  if (n != 9 || !get(o[0], &x) || !get(o[1], &a) || !get(o[2], &B) || !get(o[3], &C) || !get(o[4], &state) ||
      !get(o[5], &dt, true) || !get(o[6], &D, true) || !get(o[7], &z, true) || !get(o[8], &out, true) || !x->is_cuda() ||
      x->dim() != 3 || B->dim() != 3 || state->dim() != 4)
    Py_RETURN_NONE;
  const int dtype = dtype_of(*x);
  const int64_t b = x->size(0), h = x->size(1), p = x->size(2), g = B->size(1), ns = B->size(2);
  const auto st = x->scalar_type();
  if (dtype < 0 || g <= 0 || h % g != 0 || !inner(*x) || !inner(*B)) Py_RETURN_NONE;
  if (a->scalar_type() != at::kFloat || !shaped(*a, {b, h}) || B->scalar_type() != st || !shaped(*B, {b, g, ns}) ||
      C->scalar_type() != st || !shaped(*C, {b, g, ns}) || !inner(*C) || state->scalar_type() != at::kFloat ||
      !shaped(*state, {b, h, ns, p}) || !state->is_contiguous())
    Py_RETURN_NONE;
  if (dt->defined() && (dt->scalar_type() != st || !shaped(*dt, {b, h}))) Py_RETURN_NONE;
  if (z->defined() && (z->scalar_type() != st || !shaped(*z, {b, h, p}) || !inner(*z))) Py_RETURN_NONE;
  if (D->defined() && (!shaped(*D, {h}) || !D->is_contiguous() || (D->scalar_type() != st && D->scalar_type() != at::kFloat)))
    Py_RETURN_NONE;
  if (out->defined() && (out->scalar_type() != st || !shaped(*out, {b, h, p}) || !out->is_contiguous())) Py_RETURN_NONE;
  Where w(*x);
  if (!w.here(*a) || !w.here(*B) || !w.here(*C) || !w.here(*state) || !w.here(*dt) || !w.here(*D) || !w.here(*z) || !w.here(*out))
    Py_RETURN_NONE;
  Tensor y = out->defined() ? *out : at::empty({b, h, p}, x->options());
  SsdStepArgs s = {};
  s.x = x->data_ptr(); s.a = static_cast<const float*>(a->data_ptr()); s.B = B->data_ptr(); s.C = C->data_ptr();
  s.state = static_cast<float*>(state->data_ptr()); s.y = y.data_ptr();
  s.batch = (int)b; s.nheads = (int)h; s.headdim = (int)p; s.dstate = (int)ns; s.ngroups = (int)g; s.dtype = dtype;
  for (int d = 0; d < 2; ++d) {
    s.x_stride[d] = x->stride(d); s.a_stride[d] = a->stride(d); s.b_stride[d] = B->stride(d); s.c_stride[d] = C->stride(d);
  }
  if (dt->defined()) { s.dt = dt->data_ptr(); s.dt_stride[0] = dt->stride(0); s.dt_stride[1] = dt->stride(1); }
  if (z->defined()) { s.z = z->data_ptr(); s.z_stride[0] = z->stride(0); s.z_stride[1] = z->stride(1); }
  if (D->defined()) { s.D = D->data_ptr(); s.d_in_dtype = D->scalar_type() == st && st != at::kFloat; }
  if (const int rc = f_step(&s, w.stream())) return declined(rc);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// dt_prologue(dt_raw, dt_bias, A_log) -> (dt, A_dt)
PyObject* py_dt(PyObject*, PyObject* const* o, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Tensor *r, *bias, *al;
  if (n != 3 || !get(o[0], &r) || !get(o[1], &bias, true) || !get(o[2], &al) || !r->is_cuda() || r->dim() != 3) Py_RETURN_NONE;
  const int dtype = dtype_of(*r);
  const int64_t b = r->size(0), l = r->size(1), h = r->size(2);
  if (dtype < 0 || r->stride(2) != 1 || al->scalar_type() != at::kFloat || !shaped(*al, {h}) || !al->is_contiguous()) Py_RETURN_NONE;
  if (bias->defined() && (!shaped(*bias, {h}) || bias->scalar_type() != r->scalar_type() || !bias->is_contiguous())) Py_RETURN_NONE;
  Where w(*r);
  if (!w.here(*bias) || !w.here(*al)) Py_RETURN_NONE;
  Tensor dt = at::empty({b, l, h}, r->options());
  Tensor A = at::empty({b, l, h}, r->options().dtype(at::kFloat));
  if (const int rc = f_dt(r->data_ptr(), r->stride(0), r->stride(1), bias->defined() ? bias->data_ptr() : nullptr,
                          static_cast<const float*>(al->data_ptr()), dt.data_ptr(), static_cast<float*>(A.data_ptr()), (int)b,
                          (int)l, (int)h, dtype, w.stream()))
    return declined(rc);
  PyObject* t = PyTuple_New(2);
  if (!t) return nullptr;
  PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(std::move(dt)));
  PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(std::move(A)));
  return t;
  END_HANDLE_TH_ERRORS
}

// conv1d_silu(x, weight, bias, out) -> y
PyObject* py_conv(PyObject*, PyObject* const* o, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Tensor *x, *w, *bias, *out;
  if (n != 4 || !get(o[0], &x) || !get(o[1], &w) || !get(o[2], &bias, true) || !get(o[3], &out, true) || !x->is_cuda() || x->dim() != 3)
    Py_RETURN_NONE;
  const int dtype = dtype_of(*x);
  const int64_t b = x->size(0), l = x->size(1), d = x->size(2);
  const auto st = x->scalar_type();
  if (dtype < 0 || x->stride(2) != 1 || d <= 0 || w->scalar_type() != st || !w->is_contiguous() || w->dim() < 2 || w->size(0) != d ||
      w->numel() != d * w->size(-1))
    Py_RETURN_NONE;
  if (bias->defined() && (!shaped(*bias, {d}) || bias->scalar_type() != st || !bias->is_contiguous())) Py_RETURN_NONE;
  if (out->defined() && (out->scalar_type() != st || out->sizes() != x->sizes() || !inner(*out))) Py_RETURN_NONE;
  Where q(*x);
  if (!q.here(*w) || !q.here(*bias) || !q.here(*out)) Py_RETURN_NONE;
  Tensor y = out->defined() ? *out : at::empty({b, l, d}, x->options());
  if (const int rc = f_conv(x->data_ptr(), w->data_ptr(), bias->defined() ? bias->data_ptr() : nullptr, y.data_ptr(), (int)b,
                            (int)l, (int)d, (int)w->size(-1), dtype, x->stride(0), x->stride(1), y.stride(0), y.stride(1), q.stream()))
    return declined(rc);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// forward(X, A, B, C, chunk, dt, initial_states, D, z, out, return_final_state) -> Y or (Y, final_state)
PyObject* py_forward(PyObject*, PyObject* const* o, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Tensor *X, *A, *B, *C, *dt, *init, *D, *z, *out;
  if (n != 11 || !get(o[0], &X) || !get(o[1], &A) || !get(o[2], &B) || !get(o[3], &C) || !PyLong_CheckExact(o[4]) ||
      !get(o[5], &dt, true) || !get(o[6], &init, true) || !get(o[7], &D, true) || !get(o[8], &z, true) ||
      !get(o[9], &out, true) || !X->is_cuda() || X->dim() != 4 || A->dim() != 3 || B->dim() != 4)
    Py_RETURN_NONE;
  int over = 0;
  const long long chunk = PyLong_AsLongLongAndOverflow(o[4], &over);
  const bool want_final = o[10] == Py_True;
  const int dtype = dtype_of(*X);
  const auto st = X->scalar_type();
  const int64_t b = X->size(0), s = X->size(1), h = X->size(2), p = X->size(3), g = B->size(2), ns = B->size(3);
  if (dtype < 0 || over || chunk <= 0 || chunk > 0x7fffffff || g <= 0 || h % g != 0 || !inner(*X) || !inner(*B) ||
      A->scalar_type() != at::kFloat || !shaped(*A, {b, s, h}) || B->scalar_type() != st || !shaped(*B, {b, s, g, ns}) ||
      C->scalar_type() != st || C->sizes() != B->sizes() || !inner(*C))
    Py_RETURN_NONE;
  if (dt->defined() && (dt->scalar_type() != st || !shaped(*dt, {b, s, h}))) Py_RETURN_NONE;
  if (init->defined() && (init->scalar_type() != at::kFloat || !shaped(*init, {b, h, ns, p}) || !init->is_contiguous())) Py_RETURN_NONE;
  if (D->defined() && (!shaped(*D, {h}) || !D->is_contiguous() || (D->scalar_type() != st && D->scalar_type() != at::kFloat)))
    Py_RETURN_NONE;
  if (z->defined() && (z->scalar_type() != st || z->sizes() != X->sizes() || !inner(*z))) Py_RETURN_NONE;
  if (out->defined() && (out->scalar_type() != st || out->sizes() != X->sizes() || !inner(*out))) Py_RETURN_NONE;
  Where w(*X);
  if (!w.here(*A) || !w.here(*B) || !w.here(*C) || !w.here(*dt) || !w.here(*init) || !w.here(*D) || !w.here(*z) || !w.here(*out))
    Py_RETURN_NONE;
  Tensor Y = out->defined() ? *out : at::empty({b, s, h, p}, X->options());
  Tensor fin;
  if (want_final) fin = at::empty({b, h, ns, p}, X->options().dtype(at::kFloat));
  SsdArgs a = {};
  a.X = X->data_ptr(); a.A = static_cast<const float*>(A->data_ptr()); a.B = B->data_ptr(); a.C = C->data_ptr(); a.Y = Y.data_ptr();
  if (dt->defined()) { a.dt = dt->data_ptr(); strides3(*dt, a.dt_stride); }
  if (init->defined()) a.initial_state = static_cast<const float*>(init->data_ptr());
  if (want_final) a.final_state = static_cast<float*>(fin.data_ptr());
  if (D->defined()) {
    a.D = static_cast<const float*>(D->data_ptr());
    if (D->scalar_type() != at::kFloat) a.flags |= SSD_FLAG_D_IN_DTYPE;
  }
  if (z->defined()) { a.Z = z->data_ptr(); strides4(*z, a.z_stride); }
  a.status = static_cast<int32_t*>(status_word(w.dev.index()).data_ptr());
  a.batch = (int)b; a.seqlen = (int)s; a.nheads = (int)h; a.headdim = (int)p; a.dstate = (int)ns; a.ngroups = (int)g;
  a.chunk = (int)chunk; a.dtype = dtype;
  strides4(*X, a.x_stride); strides3(*A, a.a_stride); strides4(*B, a.b_stride); strides4(*C, a.c_stride); strides4(Y, a.y_stride);
  const size_t need = f_workspace(&a);
  Tensor ws;   // from the current stream's memory: calls on other streams have their own
  if (need) {
    ws = at::empty({(int64_t)need}, X->options().dtype(at::kByte));
    a.workspace = ws.data_ptr();
    a.workspace_bytes = need;
  }
  if (const int rc = f_forward(&a, w.stream())) return declined(rc);
  if (!want_final) return THPVariable_Wrap(std::move(Y));
  PyObject* t = PyTuple_New(2);
  if (!t) return nullptr;
  PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(std::move(Y)));
  PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(std::move(fin)));
  return t;
  END_HANDLE_TH_ERRORS
}

// workspace(device_index, bytes), status_word(device_index): the tensors that the long way uses too
PyObject* py_workspace(PyObject*, PyObject* const* o, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 2) Py_RETURN_NONE;
  const long dev = PyLong_AsLong(o[0]);
  const long long bytes = PyLong_AsLongLong(o[1]);
  if (PyErr_Occurred() || dev < 0 || dev >= kMaxDevices) return PyErr_Occurred() ? nullptr : (Py_INCREF(Py_None), Py_None);
  return THPVariable_Wrap(workspace((int)dev, bytes));
  END_HANDLE_TH_ERRORS
}
PyObject* py_status(PyObject*, PyObject* const* o, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 1) Py_RETURN_NONE;
  const long dev = PyLong_AsLong(o[0]);
  if (PyErr_Occurred() || dev < 0 || dev >= kMaxDevices) return PyErr_Occurred() ? nullptr : (Py_INCREF(Py_None), Py_None);
  return THPVariable_Wrap(status_word((int)dev));
  END_HANDLE_TH_ERRORS
}

// init(forward, workspace_bytes, step_strided, conv1d_silu, dt_prologue, raise): addresses in the loaded library, and the
// function that raises the exception of an error code
PyObject* py_init(PyObject*, PyObject* const* o, Py_ssize_t n) {
  if (n != 6) {
    PyErr_SetString(PyExc_TypeError, "init takes five addresses and a function");
    return nullptr;
  }
  void* f[5];
  for (int i = 0; i < 5; ++i) f[i] = PyLong_AsVoidPtr(o[i]);
  if (PyErr_Occurred()) return nullptr;
  f_forward = reinterpret_cast<decltype(f_forward)>(f[0]);
  f_workspace = reinterpret_cast<decltype(f_workspace)>(f[1]);
  f_step = reinterpret_cast<decltype(f_step)>(f[2]);
  f_conv = reinterpret_cast<decltype(f_conv)>(f[3]);
  f_dt = reinterpret_cast<decltype(f_dt)>(f[4]);
  Py_INCREF(o[5]);
  Py_XSETREF(f_raise, o[5]);
  Py_RETURN_NONE;
}

#define FAST(f) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(f)), METH_FASTCALL, nullptr
PyMethodDef methods[] = {{"init", FAST(py_init)}, {"step", FAST(py_step)}, {"dt_prologue", FAST(py_dt)},
                         {"conv1d_silu", FAST(py_conv)}, {"forward", FAST(py_forward)}, {"workspace", FAST(py_workspace)},
                         {"status_word", FAST(py_status)}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "ssd_b200_torch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_ssd_b200_torch(void) { return PyModule_Create(&module); }
