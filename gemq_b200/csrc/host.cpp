// Host side of the calls that a decode step makes, in native code: argument checks, output allocation, stream
// and device lookup and the library call.  In Python the same steps took 12 to 20 us a call, several times the
// kernels of a small linear.  Every function returns None when it does not take the call (a dtype, shape or
// alignment of another path, tensors on different devices, a library error): the Python wrappers then go on
// to that path or raise the error.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include "../../include/gemq_b200.h"

namespace {

using at::Tensor;

PyObject* none() { Py_RETURN_NONE; }
bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
bool half_type(const Tensor& t) { return t.scalar_type() == at::kHalf || t.scalar_type() == at::kBFloat16; }

const Tensor* tensor(PyObject* o) { return THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr; }

void* stream_of(const Tensor& x) { return c10::cuda::getCurrentCUDAStream(x.get_device()).stream(); }

Tensor empty_cuda(at::IntArrayRef sizes, at::ScalarType t, const Tensor& like) {
  return at::empty(sizes, at::TensorOptions().dtype(t).device(like.device()));
}

// plain(*args) -> whether the call is one that nobody but its caller looks at: kernels/_ops.py, plain_call, which asks
// here first.  A default device is a function mode: False, the Python form tells it from others.
PyObject* plain(PyObject*, PyObject* const* a, Py_ssize_t n) {
  const auto& tls = c10::impl::tls_local_dispatch_key_set().included_;
  if (c10::impl::TorchDispatchModeTLS::any_modes_set() || at::impl::torch_function_mode_enabled() ||
      tls.has(c10::DispatchKey::FuncTorchDynamicLayerFrontMode) || torch::jit::tracer::isTracing())
    Py_RETURN_FALSE;
  const bool grad = c10::GradMode::is_enabled();
  for (Py_ssize_t i = 0; i < n; ++i) {
    if (!THPVariable_Check(a[i])) continue;
    const Tensor* t = tensor(a[i]);
    if (!t || (grad && t->requires_grad()) || t->_fw_grad(0).defined()) Py_RETURN_FALSE;
  }
  Py_RETURN_TRUE;
}

// linear(x, w_q, scales, zeros, nbits, group_size, bias | None, err_word_ptr, mode)
// x [..., K] fp16 / bf16 -> [..., N] of the same type.  mode: the caller's contract.
enum { kLayer = 0,      // any leading dimensions
       kRowsOp = 1,     // 2-D fp16
       kOneRowOp = 2,   // [1, K] fp16
       kGemmOp = 3 };   // 2-D; below 32 rows fp16
PyObject* linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 9) { PyErr_SetString(PyExc_TypeError, "linear takes 9 arguments"); return nullptr; }
  const Tensor *x = tensor(a[0]), *w = tensor(a[1]), *s = tensor(a[2]), *z = tensor(a[3]);
  if (!x || !w || !s || !z) return none();
  const Tensor* bias = nullptr;
  if (a[6] != Py_None && !(bias = tensor(a[6]))) return none();
  const long nbits = PyLong_AsLong(a[4]), G = PyLong_AsLong(a[5]);
  int32_t* err = static_cast<int32_t*>(PyLong_AsVoidPtr(a[7]));
  if (PyErr_Occurred()) { PyErr_Clear(); return none(); }
  const long mode = PyLong_AsLong(a[8]);
  if (!err || nbits < 1 || nbits > 4 || G != 128 || x->dim() < 1 || w->dim() != 2 || s->dim() != 2 || z->dim() != 2) return none();
  if (!x->is_cuda() || !half_type(*x) || (mode != kLayer && x->dim() != 2)) return none();
  const int64_t K = x->size(-1), N = w->size(1), eps = 32 / nbits;
  if (K <= 0 || K % 128 || K > 32768 || N <= 0 || N % 32 || x->numel() == 0) return none();
  const int64_t M = x->numel() / K;
  if (M > (1 << 30) || (mode == kOneRowOp && M != 1)) return none();
  if (M == 1 && x->scalar_type() == at::kHalf && gemq_one_row_streams(static_cast<int>(N), static_cast<int>(K))) return none();
  const bool gemm = mode == kLayer ? gemq_linear_takes_gemm(static_cast<int>(M), static_cast<int>(N), static_cast<int>(K), static_cast<int>(nbits))
                                   : mode == kGemmOp && M >= 32;
  if (mode != kLayer && !gemm && x->scalar_type() != at::kHalf) return none();
  const auto dev = x->device();
  if (w->scalar_type() != at::kInt || w->size(0) != (K + eps - 1) / eps || !w->is_contiguous() || w->device() != dev) return none();
  for (const Tensor* m : {s, z})
    if (m->scalar_type() != at::kHalf || m->size(0) != K / 128 || m->size(1) != N || !m->is_contiguous() || m->device() != dev)
      return none();
  // only what works on rows of one pitch; other strides are made contiguous by the Python path
  int64_t ldx = K;
  if (x->dim() == 2) {
    if (x->stride(1) != 1) return none();
    ldx = x->stride(0);
  } else if (!x->is_contiguous()) {
    return none();
  }
  if (ldx < K || ldx > (1 << 30)) { if (M > 1) return none(); ldx = K; }
  const void* wp = w->data_ptr();
  if (!aligned16(wp) || !aligned16(s->data_ptr()) || !aligned16(z->data_ptr())) return none();
  const bool bf = x->scalar_type() == at::kBFloat16;
  Tensor b;
  if (bias) {
    if (bias->dim() != 1 || bias->size(0) != N) return none();
    b = bias->scalar_type() == x->scalar_type() && bias->device() == dev && bias->is_contiguous()
            ? *bias : bias->to(dev, x->scalar_type()).contiguous();
  }
  c10::cuda::CUDAGuard guard(dev);
  at::DimVector shape(x->sizes().begin(), x->sizes().end());
  shape.back() = N;
  Tensor y = empty_cuda(shape, x->scalar_type(), *x);
  const void* bp = bias ? b.data_ptr() : nullptr;
  int rc;
  if (gemm) {
    if (ldx != K || !aligned16(x->data_ptr())) return none();
    const size_t parts = gemq_linear_gemm_scratch_bytes(static_cast<int>(M), static_cast<int>(N), static_cast<int>(K), static_cast<int>(nbits));
    Tensor scratch;
    if (parts) scratch = empty_cuda({static_cast<int64_t>(parts / 4)}, at::kFloat, *x);
    rc = gemq_linear_gemm(x->data_ptr(), nullptr, static_cast<const int32_t*>(wp), s->data_ptr(), z->data_ptr(), nullptr, nullptr,
                          nullptr, static_cast<int>(nbits), bp, y.data_ptr(), static_cast<int>(M), static_cast<int>(N),
                          static_cast<int>(K), 128, bf, err, parts ? scratch.data_ptr() : nullptr, parts, stream_of(*x));
    if (rc) return none();
  } else {
    rc = gemq_linear_rows(x->data_ptr(), static_cast<int>(ldx), bf, static_cast<const int32_t*>(wp), s->data_ptr(), z->data_ptr(),
                          bp, y.data_ptr(), static_cast<int>(M), static_cast<int>(N), static_cast<int>(K), static_cast<int>(nbits),
                          128, err, stream_of(*x));
    if (rc) return none();
  }
  return THPVariable_Wrap(std::move(y));
}

// moe_decode(layer_ptr, x, scratch, hidden, top_k, route_mode): every row of x [..., hidden], fp16 or bf16 -> out like x
PyObject* moe_decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 6) { PyErr_SetString(PyExc_TypeError, "moe_decode takes 6 arguments"); return nullptr; }
  const auto* L = static_cast<const gemq_moe_layer_t*>(PyLong_AsVoidPtr(a[0]));
  const Tensor *x = tensor(a[1]), *sc = tensor(a[2]);
  const long D = PyLong_AsLong(a[3]), A = PyLong_AsLong(a[4]), mode = PyLong_AsLong(a[5]);
  if (PyErr_Occurred()) { PyErr_Clear(); return none(); }
  if (!L || !x || !sc || !x->is_cuda() || !half_type(*x) || x->dim() < 1 || x->size(-1) != D || x->numel() == 0) return none();
  if (!sc->is_cuda() || sc->device() != x->device()) return none();
  c10::cuda::CUDAGuard guard(x->device());
  const bool bf = x->scalar_type() == at::kBFloat16;
  Tensor xh = (bf ? x->to(at::kHalf) : *x).contiguous();
  const int64_t T = x->numel() / D;
  Tensor out = empty_cuda(x->sizes(), at::kHalf, *x);
  // routing results: not returned, but part of the call's contract
  Tensor r = empty_cuda({T * A * 10}, at::kByte, *x);
  auto* idx = static_cast<int64_t*>(r.data_ptr());
  void* w = static_cast<char*>(r.data_ptr()) + T * A * 8;
  const int rc = gemq_moe_decode(L, xh.data_ptr(), out.data_ptr(), idx, w, static_cast<int>(T), 1, static_cast<int>(mode),
                                 sc->data_ptr(), static_cast<size_t>(sc->numel()), stream_of(*x));
  if (rc) return none();
  return THPVariable_Wrap(bf ? out.to(at::kBFloat16) : out);
}

// moe_prefill(layer_ptr, x, scratch | None, hidden, top_k, n_experts, route_mode, want_logits)
// -> (out, logits | None), logits [T, E] of x's type; None also when the scratch is too small, and under capture
// (the block then keeps the scratch for the graph).
PyObject* moe_prefill(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 8) { PyErr_SetString(PyExc_TypeError, "moe_prefill takes 8 arguments"); return nullptr; }
  const auto* L = static_cast<const gemq_moe_layer_t*>(PyLong_AsVoidPtr(a[0]));
  const Tensor *x = tensor(a[1]), *sc = tensor(a[2]);
  const long D = PyLong_AsLong(a[3]), A = PyLong_AsLong(a[4]), E = PyLong_AsLong(a[5]), mode = PyLong_AsLong(a[6]);
  if (PyErr_Occurred()) { PyErr_Clear(); return none(); }
  const bool want = a[7] == Py_True;
  if (!L || !x || !sc || !x->is_cuda() || !half_type(*x) || x->dim() < 1 || x->size(-1) != D || x->numel() == 0) return none();
  if (!x->is_contiguous() || !aligned16(x->data_ptr()) || sc->device() != x->device()) return none();
  const int64_t T = x->numel() / D;
  if (T > (1 << 24) || gemq_moe_prefill_scratch_bytes(L, static_cast<int>(T)) > static_cast<size_t>(sc->numel())) return none();
  c10::cuda::CUDAGuard guard(x->device());
  if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) return none();
  Tensor out = empty_cuda(x->sizes(), x->scalar_type(), *x);
  Tensor logits;
  if (want) logits = empty_cuda({T, E}, x->scalar_type(), *x);
  Tensor r = empty_cuda({T * A * 10}, at::kByte, *x);
  auto* idx = static_cast<int64_t*>(r.data_ptr());
  void* w = static_cast<char*>(r.data_ptr()) + T * A * 8;
  const int rc = gemq_moe_prefill(L, x->data_ptr(), out.data_ptr(), idx, w, want ? logits.data_ptr() : nullptr,
                                  static_cast<int>(T), 2, static_cast<int>(mode), x->scalar_type() == at::kBFloat16, sc->data_ptr(),
                                  static_cast<size_t>(sc->numel()), stream_of(*x));
  if (rc) return none();
  PyObject* o = THPVariable_Wrap(std::move(out));
  PyObject* l = want ? THPVariable_Wrap(std::move(logits)) : none();
  PyObject* t = PyTuple_Pack(2, o, l);
  Py_DECREF(o);
  Py_DECREF(l);
  return t;
}

template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  return F(self, a, n);
  END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"plain", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&guarded<plain>)), METH_FASTCALL, nullptr},
    {"linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&guarded<linear>)), METH_FASTCALL, nullptr},
    {"moe_decode", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&guarded<moe_decode>)), METH_FASTCALL, nullptr},
    {"moe_prefill", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&guarded<moe_prefill>)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) { return PyModule_Create(&module); }
