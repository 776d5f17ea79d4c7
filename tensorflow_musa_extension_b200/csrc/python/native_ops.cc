// Native host path of the ops: argument checks, output and scratch allocation
// and the launcher call of one op in one C++ function.
//
// A FusedBatchNormV3 + FusedBatchNormGradV3 pair cost 85 us of host time in
// Python (30 attribute reads, 13 tensor allocations, two context managers,
// ctypes conversions of 18 arguments) for 19 us of device work on [8,14,14,64],
// 25 us here with every tensor allocated through the dispatcher and 15 without; the
// functions here take the calls that need no conversion - strided, contiguous
// tensors of the right types on one CUDA device - and return None for every other
// call, which the Python path then converts or refuses as it always did.  So what
// is accepted, refused and returned does not depend on this file.
//
// Scratch comes from the caching allocator for the length of the call: it is
// ordered by the current stream, private to the call (several threads may run
// on one stream) and recorded by a graph capture like any other allocation.
#include <dlfcn.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <ATen/ATen.h>
#include <ATen/EmptyTensor.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <cmath>

#include "../../../include/musa_plugin_kernels.h"

namespace {

// Launchers of the kernel library that the loader opened.
struct Api {
#define MUSA_API(X)                                                                       \
  X(BnWorkspaceBytes) X(LaunchBnFwdTrainOp) X(LaunchBnFwdInferOp) X(LaunchBnGradOp)       \
  X(LaunchBiasAct_F32) X(LaunchBiasAct_F16) X(LaunchBiasAct_BF16)                         \
  X(BiasGradWorkspaceBytes) X(LaunchBiasAddReluGrad_F32) X(LaunchBiasAddReluGrad_F16)     \
  X(LaunchBiasAddReluGrad_BF16) X(LaunchLayerNorm_F32) X(LaunchLayerNorm_F16)             \
  X(LaunchLayerNorm_BF16) X(LayerNormGradWorkspaceBytes) X(LaunchLayerNormGrad_F32)       \
  X(LaunchLayerNormGrad_F16) X(LaunchLayerNormGrad_BF16) X(LaunchRmsNormFloat)            \
  X(LaunchRmsNormBFloat16) X(LaunchRmsNormGradDxFloat) X(LaunchRmsNormGradDxBFloat16)     \
  X(LaunchApplyAdamGroupHostTable)
#define X(name) decltype(&::name) name = nullptr;
  MUSA_API(X)
#undef X
};
Api g_api;

// dtype code of the launchers (MUSA_DT_*), or -1.
int DtypeCode(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return MUSA_DT_F32;
    case at::kHalf: return MUSA_DT_F16;
    case at::kBFloat16: return MUSA_DT_BF16;
    default: return -1;
  }
}

template <typename F>
F ByDtype(int code, F f32, F f16, F bf16) {
  return code == MUSA_DT_F32 ? f32 : code == MUSA_DT_F16 ? f16 : bf16;
}

// The tensor behind `obj` if the launchers can take it as it is: a plain
// torch.Tensor or Parameter (no subclass, no transform wrapper, no lazy
// conjugate), contiguous, on a CUDA device.
const at::Tensor* Direct(PyObject* obj) {
  if (!THPVariable_CheckExact(obj)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(obj);
  static const c10::DispatchKeySet kWrapped =
      c10::DispatchKeySet({c10::DispatchKey::Python, c10::DispatchKey::PythonTLSSnapshot,
                           c10::DispatchKey::FuncTorchBatched,
                           c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Batched,
                           c10::DispatchKey::Functionalize, c10::DispatchKey::Conjugate,
                           c10::DispatchKey::Negative, c10::DispatchKey::ZeroTensor});
  if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided) return nullptr;
  if (t.key_set().has_any(kWrapped) || !t.is_contiguous()) return nullptr;
  return &t;
}

// No mode that wants to see the calls is active.
bool NoModes() {
  return !c10::impl::TorchDispatchModeTLS::any_modes_set() &&
         at::impl::PythonTorchFunctionTLS::stack_len() == 0;
}

bool IsF32Vector(const at::Tensor* t, int64_t c, const at::Tensor& like) {
  return t != nullptr && t->scalar_type() == at::kFloat && t->dim() == 1 && t->numel() == c &&
         t->device() == like.device();
}

// Outputs and scratch come from torch's caching allocator on the current device and
// stream, without the dispatcher's way there: it has nothing left to decide for a
// plain CUDA tensor.
constexpr c10::DispatchKeySet kCudaKey(c10::DispatchKey::CUDA);

c10::Allocator* Allocator() { return c10::cuda::CUDACachingAllocator::get(); }

at::Tensor EmptyLike(const at::Tensor& t) {
  if (t.has_names()) return at::empty_like(t);
  return at::detail::empty_strided_generic(t.sizes(), t.strides(), Allocator(), kCudaKey,
                                           t.scalar_type());
}

at::Tensor Empty(at::IntArrayRef sizes, at::ScalarType dtype) {
  return at::detail::empty_generic(sizes, Allocator(), kCudaKey, dtype, std::nullopt);
}

// A per-channel output.  Every one has a storage of its own, as the Python path's do: a caller
// may resize, save or keep one without touching or holding the others.
at::Tensor Vector(int64_t c) { return Empty(c, at::kFloat); }

// Scratch of at least `bytes`, for the length of the call.
struct Scratch {
  explicit Scratch(size_t bytes)
      : size(bytes < 16 ? 16 : bytes), data(Allocator()->allocate(size)) {}
  size_t size;
  c10::DataPtr data;
};

// [outer, channels, inner] of a shape; false: not a layout name or too few axes.
bool Geometry(const at::Tensor& x, PyObject* format, int64_t* outer, int64_t* c, int64_t* inner) {
  if (!PyUnicode_Check(format) || x.dim() < 2) return false;
  const auto sizes = x.sizes();
  if (PyUnicode_CompareWithASCIIString(format, "NHWC") == 0) {
    *c = sizes[x.dim() - 1];
    *inner = 1;
    *outer = 1;
    for (int64_t i = 0; i + 1 < x.dim(); ++i) *outer *= sizes[i];
    return true;
  }
  if (PyUnicode_CompareWithASCIIString(format, "NCHW") == 0) {
    *outer = sizes[0];
    *c = sizes[1];
    *inner = 1;
    for (int64_t i = 2; i < x.dim(); ++i) *inner *= sizes[i];
    return true;
  }
  return false;
}

// Host scalars: Python floats and ints only (float() of anything else is the
// Python path's business).
bool Number(PyObject* o, double* out) {
  if (PyFloat_CheckExact(o)) {
    *out = PyFloat_AS_DOUBLE(o);
    return true;
  }
  if (PyLong_CheckExact(o)) {
    *out = PyLong_AsDouble(o);
    if (*out == -1.0 && PyErr_Occurred()) {
      PyErr_Clear();
      return false;
    }
    return true;
  }
  return false;
}

bool Flag(PyObject* o, bool* out) {
  if (!PyBool_Check(o)) return false;
  *out = o == Py_True;
  return true;
}

// The tensors as a tuple, or the launcher's error code as an int.
PyObject* Results(int rc, std::initializer_list<at::Tensor> tensors) {
  if (rc != 0) return PyLong_FromLong(rc);
  PyObject* out = PyTuple_New(static_cast<Py_ssize_t>(tensors.size()));
  if (out == nullptr) return nullptr;
  Py_ssize_t i = 0;
  for (const at::Tensor& t : tensors) {
    PyObject* w = THPVariable_Wrap(t);
    if (w == nullptr) {
      Py_DECREF(out);
      return nullptr;
    }
    PyTuple_SET_ITEM(out, i++, w);
  }
  return out;
}

cudaStream_t StreamOf(const at::Tensor& t) {
  return c10::cuda::getCurrentCUDAStream(t.device().index()).stream();
}

// x, scale, offset, mean, variance, epsilon, exponential_avg_factor,
// data_format, is_training
PyObject* BnForward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 9 || !NoModes()) Py_RETURN_NONE;
  const at::Tensor *xp = Direct(a[0]), *scale = Direct(a[1]), *offset = Direct(a[2]);
  const at::Tensor *mean = Direct(a[3]), *var = Direct(a[4]);
  double eps, factor;
  bool training;
  int64_t outer, c, inner;
  if (!xp || !Number(a[5], &eps) || !Number(a[6], &factor) || !Flag(a[8], &training)) {
    Py_RETURN_NONE;
  }
  const at::Tensor& x = *xp;
  const int code = DtypeCode(x.scalar_type());
  if (code < 0 || x.numel() == 0 || !Geometry(x, a[7], &outer, &c, &inner)) Py_RETURN_NONE;
  if (!IsF32Vector(scale, c, x) || !IsF32Vector(offset, c, x)) Py_RETURN_NONE;
  bool have_est = IsF32Vector(mean, c, x) && IsF32Vector(var, c, x);
  if (!have_est) {
    // Empty estimates are what a first training step passes.
    if (!training || factor != 1.0 || !IsF32Vector(mean, 0, x) || !IsF32Vector(var, 0, x)) {
      Py_RETURN_NONE;
    }
  }
  const c10::cuda::CUDAGuard guard(x.device());
  at::Tensor y = EmptyLike(x);
  at::Tensor s0 = Vector(c), s1 = Vector(c), s2 = Vector(c), s3 = Vector(c);
  at::Tensor r3 = Empty({}, at::kFloat);
  const auto F = [](const at::Tensor& t) { return static_cast<float*>(t.data_ptr()); };
  int rc;
  if (training) {
    const Scratch ws(g_api.BnWorkspaceBytes(outer, c, inner));
    pybind11::gil_scoped_release nogil;
    rc = g_api.LaunchBnFwdTrainOp(
        code, x.data_ptr(), F(*scale), F(*offset), have_est ? F(*mean) : nullptr,
        have_est ? F(*var) : nullptr, y.data_ptr(), F(s0), F(s1), F(s2), F(s3), F(r3), outer, c,
        inner, static_cast<float>(eps), static_cast<float>(factor), ws.data.get(), ws.size,
        StreamOf(x));
  } else {
    pybind11::gil_scoped_release nogil;
    rc = g_api.LaunchBnFwdInferOp(code, x.data_ptr(), F(*scale), F(*offset), F(*mean), F(*var),
                                  y.data_ptr(), F(s0), F(s1), F(s2), F(s3), F(r3), outer, c,
                                  inner, static_cast<float>(eps), StreamOf(x));
  }
  return Results(rc, {y, s0, s1, s2, s3, r3});
  END_HANDLE_TH_ERRORS
}

// dy, x, scale, mean, variance, epsilon, data_format, is_training
PyObject* BnGradient(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 8 || !NoModes()) Py_RETURN_NONE;
  const at::Tensor *dyp = Direct(a[0]), *xp = Direct(a[1]), *scale = Direct(a[2]);
  const at::Tensor *mean = Direct(a[3]), *var = Direct(a[4]);
  double eps;
  bool training;
  int64_t outer, c, inner;
  if (!dyp || !xp || !Number(a[5], &eps) || !Flag(a[7], &training)) Py_RETURN_NONE;
  const at::Tensor &x = *xp, &dy = *dyp;
  const int code = DtypeCode(x.scalar_type());
  if (code < 0 || x.numel() == 0 || !Geometry(x, a[6], &outer, &c, &inner)) Py_RETURN_NONE;
  if (dy.scalar_type() != x.scalar_type() || dy.sizes() != x.sizes() ||
      dy.device() != x.device()) {
    Py_RETURN_NONE;
  }
  if (!IsF32Vector(scale, c, x) || !IsF32Vector(mean, c, x) || !IsF32Vector(var, c, x)) {
    Py_RETURN_NONE;
  }
  const c10::cuda::CUDAGuard guard(x.device());
  at::Tensor dx = EmptyLike(x);
  at::Tensor ds = Vector(c), db = Vector(c), r4 = Vector(c), r5 = Vector(c);
  const auto F = [](const at::Tensor& t) { return static_cast<float*>(t.data_ptr()); };
  int rc;
  {
    const Scratch ws(g_api.BnWorkspaceBytes(outer, c, inner));
    pybind11::gil_scoped_release nogil;
    rc = g_api.LaunchBnGradOp(code, dy.data_ptr(), x.data_ptr(), F(*scale), F(*mean), F(*var),
                              dx.data_ptr(), F(ds), F(db), F(r4), F(r5), outer, c, inner,
                              static_cast<float>(eps), training, ws.data.get(), ws.size,
                              StreamOf(x));
  }
  return Results(rc, {dx, ds, db, r4, r5});
  END_HANDLE_TH_ERRORS
}

// value, bias, data_format, act -> y (float, half, bfloat16)
PyObject* BiasAct(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 4 || !NoModes() || !PyLong_CheckExact(a[3])) Py_RETURN_NONE;
  const at::Tensor *xp = Direct(a[0]), *b = Direct(a[1]);
  int64_t outer, c, inner;
  if (!xp || !b) Py_RETURN_NONE;
  const at::Tensor& x = *xp;
  const int code = DtypeCode(x.scalar_type());
  if (code < 0 || x.numel() == 0 || !Geometry(x, a[2], &outer, &c, &inner)) Py_RETURN_NONE;
  if (b->scalar_type() != x.scalar_type() || b->dim() != 1 || b->numel() != c ||
      b->device() != x.device()) {
    Py_RETURN_NONE;
  }
  const int act = static_cast<int>(PyLong_AsLong(a[3]));
  const c10::cuda::CUDAGuard guard(x.device());
  at::Tensor y = EmptyLike(x);
  int rc;
  {
    pybind11::gil_scoped_release nogil;
    rc = ByDtype(code, g_api.LaunchBiasAct_F32, g_api.LaunchBiasAct_F16,
                 g_api.LaunchBiasAct_BF16)(x.data_ptr(), b->data_ptr(), y.data_ptr(), outer, c,
                                           inner, act, StreamOf(x));
  }
  return Results(rc, {y});
  END_HANDLE_TH_ERRORS
}

// gradients, features, data_format -> backprops, bias_grad
PyObject* BiasReluGrad(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 3 || !NoModes()) Py_RETURN_NONE;
  const at::Tensor *gp = Direct(a[0]), *fp = Direct(a[1]);
  int64_t outer, c, inner;
  if (!gp || !fp) Py_RETURN_NONE;
  const at::Tensor &g = *gp, &f = *fp;
  const int code = DtypeCode(g.scalar_type());
  if (code < 0 || g.numel() == 0 || f.scalar_type() != g.scalar_type() ||
      f.sizes() != g.sizes() || f.device() != g.device() ||
      !Geometry(g, a[2], &outer, &c, &inner)) {
    Py_RETURN_NONE;
  }
  const c10::cuda::CUDAGuard guard(g.device());
  at::Tensor dx = EmptyLike(g);
  at::Tensor db = Empty(c, g.scalar_type());
  int rc;
  {
    const Scratch ws(
        g_api.BiasGradWorkspaceBytes(outer, c, inner, static_cast<int>(g.element_size())));
    pybind11::gil_scoped_release nogil;
    rc = ByDtype(code, g_api.LaunchBiasAddReluGrad_F32, g_api.LaunchBiasAddReluGrad_F16,
                 g_api.LaunchBiasAddReluGrad_BF16)(
        g.data_ptr(), f.data_ptr(), dx.data_ptr(), db.data_ptr(), outer, c, inner, ws.data.get(),
        ws.size, StreamOf(g));
  }
  return Results(rc, {dx, db});
  END_HANDLE_TH_ERRORS
}

// A row vector (gamma, beta) of x's type, in any shape with `last` elements.
bool RowVector(const at::Tensor* v, const at::Tensor& x, int64_t last) {
  return v != nullptr && v->scalar_type() == x.scalar_type() && v->numel() == last &&
         v->device() == x.device();
}

// x, gamma, beta, epsilon -> y
PyObject* LayerNorm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 4 || !NoModes()) Py_RETURN_NONE;
  const at::Tensor *xp = Direct(a[0]), *g = Direct(a[1]), *b = Direct(a[2]);
  double eps;
  if (!xp || !Number(a[3], &eps) || xp->dim() < 1 || xp->numel() == 0) Py_RETURN_NONE;
  const at::Tensor& x = *xp;
  const int code = DtypeCode(x.scalar_type());
  const int64_t last = x.size(-1);
  if (code < 0 || !RowVector(g, x, last) || !RowVector(b, x, last)) Py_RETURN_NONE;
  const c10::cuda::CUDAGuard guard(x.device());
  at::Tensor y = EmptyLike(x);
  int rc;
  {
    pybind11::gil_scoped_release nogil;
    rc = ByDtype(code, g_api.LaunchLayerNorm_F32, g_api.LaunchLayerNorm_F16,
                 g_api.LaunchLayerNorm_BF16)(x.data_ptr(), g->data_ptr(), b->data_ptr(),
                                             y.data_ptr(), nullptr, nullptr, x.numel() / last,
                                             last, static_cast<float>(eps), StreamOf(x));
  }
  return Results(rc, {y});
  END_HANDLE_TH_ERRORS
}

// dy, x, gamma, beta, epsilon -> dx, dgamma, dbeta
PyObject* LayerNormGrad(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 5 || !NoModes()) Py_RETURN_NONE;
  const at::Tensor *dp = Direct(a[0]), *xp = Direct(a[1]), *g = Direct(a[2]), *b = Direct(a[3]);
  double eps;
  if (!dp || !xp || !Number(a[4], &eps) || xp->dim() < 1 || xp->numel() == 0) Py_RETURN_NONE;
  const at::Tensor &x = *xp, &dy = *dp;
  const int code = DtypeCode(x.scalar_type());
  const int64_t last = x.size(-1);
  if (code < 0 || dy.scalar_type() != x.scalar_type() || dy.sizes() != x.sizes() ||
      dy.device() != x.device() || !RowVector(g, x, last) || !RowVector(b, x, last)) {
    Py_RETURN_NONE;
  }
  const c10::cuda::CUDAGuard guard(x.device());
  at::Tensor dx = EmptyLike(x), dg = EmptyLike(*g), db = EmptyLike(*b);
  const int64_t rows = x.numel() / last;
  int rc;
  {
    const Scratch ws(g_api.LayerNormGradWorkspaceBytes(rows, last));
    pybind11::gil_scoped_release nogil;
    rc = ByDtype(code, g_api.LaunchLayerNormGrad_F32, g_api.LaunchLayerNormGrad_F16,
                 g_api.LaunchLayerNormGrad_BF16)(
        dy.data_ptr(), x.data_ptr(), g->data_ptr(), dx.data_ptr(), dg.data_ptr(), db.data_ptr(),
        rows, last, static_cast<float>(eps), ws.data.get(), ws.size, StreamOf(x));
  }
  return Results(rc, {dx, dg, db});
  END_HANDLE_TH_ERRORS
}

// x, gamma, epsilon -> y, normalized, inv_rms
PyObject* RmsNorm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 3 || !NoModes()) Py_RETURN_NONE;
  const at::Tensor *xp = Direct(a[0]), *g = Direct(a[1]);
  double eps;
  if (!xp || !Number(a[2], &eps) || xp->dim() < 1 || xp->numel() == 0) Py_RETURN_NONE;
  const at::Tensor& x = *xp;
  const bool f32 = x.scalar_type() == at::kFloat;
  const int64_t last = x.size(-1);
  if ((!f32 && x.scalar_type() != at::kBFloat16) || !RowVector(g, x, last)) Py_RETURN_NONE;
  const c10::cuda::CUDAGuard guard(x.device());
  at::Tensor y = EmptyLike(x), normalized = EmptyLike(x);
  auto shape = x.sizes().vec();
  shape.back() = 1;
  at::Tensor inv = Empty(shape, x.scalar_type());
  const int64_t rows = x.numel() / last;
  {
    pybind11::gil_scoped_release nogil;
    if (f32) {
      g_api.LaunchRmsNormFloat(static_cast<const float*>(x.data_ptr()),
                               static_cast<const float*>(g->data_ptr()),
                               static_cast<float*>(y.data_ptr()),
                               static_cast<float*>(normalized.data_ptr()),
                               static_cast<float*>(inv.data_ptr()), rows, last,
                               static_cast<float>(eps), StreamOf(x));
    } else {
      g_api.LaunchRmsNormBFloat16(x.data_ptr(), g->data_ptr(), y.data_ptr(),
                                  normalized.data_ptr(), inv.data_ptr(), rows, last,
                                  static_cast<float>(eps), StreamOf(x));
    }
  }
  return Results(0, {y, normalized, inv});
  END_HANDLE_TH_ERRORS
}

// x, inv_rms, gamma, dy -> dx
PyObject* RmsNormGradDx(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 4 || !NoModes()) Py_RETURN_NONE;
  const at::Tensor *xp = Direct(a[0]), *inv = Direct(a[1]), *g = Direct(a[2]), *dp = Direct(a[3]);
  if (!xp || !inv || !g || !dp || xp->numel() == 0 || g->dim() != 1) Py_RETURN_NONE;
  const at::Tensor &x = *xp, &dy = *dp;
  const bool f32 = x.scalar_type() == at::kFloat;
  const int64_t last = g->numel();
  if ((!f32 && x.scalar_type() != at::kBFloat16) || last <= 0 || x.numel() % last != 0 ||
      !RowVector(g, x, last) || !RowVector(inv, x, x.numel() / last) ||
      dy.scalar_type() != x.scalar_type() || dy.sizes() != x.sizes() ||
      dy.device() != x.device()) {
    Py_RETURN_NONE;
  }
  const c10::cuda::CUDAGuard guard(x.device());
  at::Tensor dx = EmptyLike(x);
  const int64_t rows = x.numel() / last;
  {
    pybind11::gil_scoped_release nogil;
    if (f32) {
      g_api.LaunchRmsNormGradDxFloat(static_cast<const float*>(x.data_ptr()),
                                     static_cast<const float*>(inv->data_ptr()),
                                     static_cast<const float*>(g->data_ptr()),
                                     static_cast<const float*>(dy.data_ptr()),
                                     static_cast<float*>(dx.data_ptr()), rows, last, StreamOf(x));
    } else {
      g_api.LaunchRmsNormGradDxBFloat16(x.data_ptr(), inv->data_ptr(), g->data_ptr(),
                                        dy.data_ptr(), dx.data_ptr(), rows, last, StreamOf(x));
    }
  }
  return Results(0, {dx});
  END_HANDLE_TH_ERRORS
}

// var, m, v, grad -> (device index, state code, grad code) as one number, or
// -1: whether the update can share a launch with its neighbours.
int AdamKind(PyObject* const* a) {
  const at::Tensor *t = Direct(a[0]), *m = Direct(a[1]), *v = Direct(a[2]), *g = Direct(a[3]);
  if (!t || !m || !v || !g) return -1;
  const int state = DtypeCode(t->scalar_type()), grad = DtypeCode(g->scalar_type());
  if (state < 0 || grad < 0 || (state != MUSA_DT_F32 && grad != state)) return -1;
  if (m->scalar_type() != t->scalar_type() || v->scalar_type() != t->scalar_type()) return -1;
  if (g->device() != t->device() || m->device() != t->device() || v->device() != t->device()) {
    return -1;
  }
  if (t->sizes() != g->sizes() || t->sizes() != m->sizes() || t->sizes() != v->sizes()) return -1;
  return (t->device().index() * 4 + state) * 4 + grad;
}

PyObject* AdamKindOf(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  return PyLong_FromLong(n == 4 && NoModes() ? AdamKind(a) : -1);
  END_HANDLE_TH_ERRORS
}

// list of (var, m, v, grad) tuples of one kind, alpha, beta1, beta2, epsilon,
// use_nesterov -> launcher code
PyObject* AdamGroup(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 6 || !PyList_CheckExact(a[0])) Py_RETURN_NONE;
  double alpha, b1, b2, eps;
  bool nesterov;
  if (!Number(a[1], &alpha) || !Number(a[2], &b1) || !Number(a[3], &b2) || !Number(a[4], &eps) ||
      !Flag(a[5], &nesterov)) {
    Py_RETURN_NONE;
  }
  const Py_ssize_t count = PyList_GET_SIZE(a[0]);
  if (count == 0) return PyLong_FromLong(0);
  std::vector<void*> table[4];
  std::vector<int64_t> sizes;
  const at::Tensor *first = nullptr, *first_grad = nullptr;
  for (Py_ssize_t i = 0; i < count; ++i) {
    PyObject* q = PyList_GET_ITEM(a[0], i);
    if (!PyTuple_CheckExact(q) || PyTuple_GET_SIZE(q) != 4) Py_RETURN_NONE;
    for (int k = 0; k < 4; ++k) {
      const at::Tensor* t = Direct(PyTuple_GET_ITEM(q, k));
      if (t == nullptr) Py_RETURN_NONE;
      table[k].push_back(t->data_ptr());
      if (k == 0) {
        sizes.push_back(t->numel());
        if (i == 0) first = t;
      } else if (k == 3 && i == 0) {
        first_grad = t;
      }
    }
  }
  const c10::cuda::CUDAGuard guard(first->device());
  int rc;
  {
    pybind11::gil_scoped_release nogil;
    rc = g_api.LaunchApplyAdamGroupHostTable(
        DtypeCode(first->scalar_type()), DtypeCode(first_grad->scalar_type()), table[0].data(),
        table[1].data(), table[2].data(),
        reinterpret_cast<const void* const*>(table[3].data()), sizes.data(),
        static_cast<int>(count), static_cast<float>(alpha), static_cast<float>(b1),
        static_cast<float>(b2), static_cast<float>(eps), nesterov, StreamOf(*first));
  }
  return PyLong_FromLong(rc);
  END_HANDLE_TH_ERRORS
}

// bind(handle): the dlopen handle of the kernel library.
PyObject* Bind(PyObject*, PyObject* arg) {
  void* handle = PyLong_AsVoidPtr(arg);
  if (handle == nullptr && PyErr_Occurred()) return nullptr;
  Api api;
#define X(name)                                                                      \
  api.name = reinterpret_cast<decltype(api.name)>(dlsym(handle, #name));             \
  if (api.name == nullptr) {                                                         \
    PyErr_SetString(PyExc_AttributeError, "kernel library lacks the symbol " #name); \
    return nullptr;                                                                  \
  }
  MUSA_API(X)
#undef X
  g_api = api;
  Py_RETURN_NONE;
}

template <typename F>
PyCFunction Fast(F f) {
  return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f));
}

PyMethodDef kMethods[] = {
    {"bind", Bind, METH_O, nullptr},
    {"bn_forward", Fast(BnForward), METH_FASTCALL, nullptr},
    {"bn_gradient", Fast(BnGradient), METH_FASTCALL, nullptr},
    {"bias_act", Fast(BiasAct), METH_FASTCALL, nullptr},
    {"bias_relu_grad", Fast(BiasReluGrad), METH_FASTCALL, nullptr},
    {"layer_norm", Fast(LayerNorm), METH_FASTCALL, nullptr},
    {"layer_norm_grad", Fast(LayerNormGrad), METH_FASTCALL, nullptr},
    {"rms_norm", Fast(RmsNorm), METH_FASTCALL, nullptr},
    {"rms_norm_grad_dx", Fast(RmsNormGradDx), METH_FASTCALL, nullptr},
    {"adam_kind", Fast(AdamKindOf), METH_FASTCALL, nullptr},
    {"adam_group", Fast(AdamGroup), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_native_ops",
                       "Native host path of the ops (see raw_ops).", -1, kMethods};

}  // namespace

PyMODINIT_FUNC PyInit__native_ops() { return PyModule_Create(&kModule); }
