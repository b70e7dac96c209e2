// Native host path of the operators: argument checks, allocation of outputs and scratch, the launch
// through the C ABI and the autograd node, without Python between them.  The operators' kernels take tens
// of microseconds at small sizes, about what the same steps cost in Python for each direction.
//
// Only plain calls are served (CUDA tensors of one dtype the kernels take, shapes that agree, unit
// inner strides, no tracing and no forward-mode tangents: a tracer would record the empty output alone, and a
// tangent would be dropped without a word).  For anything else an entry returns None and the Python operators take the call: they
// convert what can be converted and raise what has to be raised.  Nothing is decided differently here.
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <atomic>
#include <cstdlib>
#include <mutex>
#include <stdexcept>

#include "../../include/splinekv_b200.h"

namespace {

using at::Tensor;

// What a kernel ORs into when a bounded wait runs out: one int32 per device, never freed (the process
// may exit after the CUDA context is gone).
constexpr int kMaxDevices = 64;
std::atomic<Tensor*> g_status[kMaxDevices];
std::mutex g_status_mu;

Tensor& status_word(int dev) {
  TORCH_CHECK(dev >= 0 && dev < kMaxDevices, "device index out of range");
  Tensor* t = g_status[dev].load(std::memory_order_acquire);
  if (!t) {
    std::lock_guard<std::mutex> lock(g_status_mu);
    t = g_status[dev].load(std::memory_order_relaxed);
    if (!t) {
      t = new Tensor(at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::Device(at::kCUDA, dev))));
      g_status[dev].store(t, std::memory_order_release);
    }
  }
  return *t;
}

[[noreturn]] void fail(int code) {
  throw std::runtime_error("splinekv_b200 error " + std::to_string(code) + ": " + skv_error_string(code));
}

bool aligned16(const void* p, int64_t stride_bytes) {
  return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && stride_bytes % 16 == 0;
}

Tensor scratch_for(size_t bytes, const Tensor& like) {
  return bytes ? at::empty({(int64_t)bytes}, like.options().dtype(at::kByte).requires_grad(false)) : Tensor();
}

// The call's problem, or false when the Python operator has to look at it.
bool plain_problem(const Tensor& z, const Tensor& C, double lo, double hi, long G, long act, double lam, long impl,
                   long order, skv_problem* p) {
  if (!z.defined() || !C.defined() || !z.is_cuda() || !C.is_cuda() || z.device() != C.device()) return false;
  if (z.unsafeGetTensorImpl()->is_python_dispatch() || C.unsafeGetTensorImpl()->is_python_dispatch()) return false;
  const auto dt = z.scalar_type();
  if ((dt != at::kBFloat16 && dt != at::kFloat) || C.scalar_type() != dt) return false;
  if (z.dim() != 2 || C.dim() != 3 || !C.is_contiguous() || z.is_conj() || z.is_neg() || C.is_neg()) return false;
  if (z.stride(1) != 1 || z.stride(0) < z.size(1)) return false;
  if (z._fw_grad(0).defined() || C._fw_grad(0).defined() || torch::jit::tracer::isTracing()) return false;
  if (C.size(0) != z.size(1) || (order != 1 && order != 2) || C.size(1) != G + order || !(hi > lo)) return false;
  if (z.size(1) > (1 << 24) || C.size(1) > 4096 || C.size(2) > 256 || C.size(2) < 1) return false;
  *p = skv_problem{};
  p->N = z.size(0);
  p->h = (int32_t)z.size(1);
  p->L = (int32_t)C.size(1);
  p->r = (int32_t)C.size(2);
  p->grid_lo = (float)lo;
  p->scale = (float)((double)G / (hi - lo));
  p->lambda_scale = (float)lam;
  p->activation = (int32_t)act;
  p->dtype = dt == at::kBFloat16 ? SKV_BF16 : SKV_F32;
  p->impl = (int32_t)impl;
  p->spline_order = (int32_t)order;
  return true;
}

// A large bf16 problem on the CUDA-core kernels: the Python operator warns about it.
bool slow_family(const skv_problem& p, bool aligned) {
  if (p.dtype != SKV_BF16 || p.impl != SKV_IMPL_AUTO || p.N * (int64_t)p.h < (1 << 24)) return false;
  return !aligned || skv_resolve_impl(&p) != SKV_IMPL_TCGEN05;
}

// [phi(z); lambda*delta] (with_base) or lambda*delta; an undefined tensor when Python has to take it.
Tensor forward(const Tensor& z, const Tensor& C, const skv_problem& p, bool with_base) {
  const int64_t width = with_base ? (int64_t)p.h + p.r : p.r;
  c10::cuda::CUDAGuard guard(z.device());
  Tensor f = at::empty({p.N, width}, z.options().requires_grad(false));
  const int64_t esz = f.element_size();
  char* base = static_cast<char*>(f.data_ptr());
  void* delta = base + (with_base ? p.h * esz : 0);
  if (slow_family(p, p.h % 8 || p.r % 8 ||
                         (aligned16(z.data_ptr(), z.stride(0) * esz) && (!with_base || aligned16(base, width * esz)))))
    return Tensor();
  const size_t need = skv_scratch_bytes(&p, SKV_OP_FORWARD);
  Tensor scratch = scratch_for(need, z);
  const int code = skv_feature_forward(&p, z.data_ptr(), z.stride(0), C.data_ptr(), with_base ? base : nullptr, width,
                                       delta, width, need ? scratch.data_ptr() : nullptr, need,
                                       static_cast<int32_t*>(status_word(z.device().index()).data_ptr()),
                                       c10::cuda::getCurrentCUDAStream(z.device().index()).stream());
  if (code) fail(code);
  return f;
}

// Autograd node of one forward (either operator): dz and dC in the dtype of z.
struct SplineFeatureBackward : public torch::autograd::Node {
  torch::autograd::SavedVariable z_, C_;
  skv_problem p{};
  bool with_base = true;

  std::string name() const override { return with_base ? "FlashSplineFeatureBackward" : "FlashSplineDeltaBackward"; }
  void release_variables() override {
    z_.reset_data();
    C_.reset_data();
  }

  torch::autograd::variable_list apply(torch::autograd::variable_list&& grads) override {
    torch::autograd::variable_list out(2);
    if (!grads[0].defined()) return out;
    at::NoGradGuard no_grad;
    Tensor z = z_.unpack(shared_from_this());
    const Tensor C = C_.unpack(shared_from_this());
    // a saved-tensor hook may hand back other strides or another dtype than it was given
    TORCH_CHECK(z.is_cuda() && C.device() == z.device(), "CUDA-only: the saved z and C must be on one CUDA device");
    TORCH_CHECK(z.dim() == 2 && z.size(0) == p.N && z.size(1) == p.h && C.dim() == 3 && C.size(0) == p.h &&
                C.size(1) == p.L && C.size(2) == p.r, "the saved z or C has another shape than the forward's");
    const auto dt = p.dtype == SKV_F32 ? at::kFloat : at::kBFloat16;
    if (z.scalar_type() != dt) z = z.to(dt);
    if (z.stride(1) != 1 || z.stride(0) < z.size(1)) z = z.contiguous();
    const Tensor table = (C.scalar_type() != dt ? C.to(dt) : C).contiguous();
    const bool need_dz = task_should_compute_output(0), need_dC = task_should_compute_output(1);
    const int64_t width = with_base ? (int64_t)p.h + p.r : p.r;
    c10::cuda::CUDAGuard guard(z.device());
    Tensor go = grads[0];
    TORCH_CHECK(go.dim() == 2 && go.size(0) == p.N && go.size(1) == width, "grad_out must be [", p.N, ", ", width,
                "], got ", go.sizes());
    if (go.scalar_type() != z.scalar_type()) go = go.to(z.scalar_type());
    if (go.stride(1) != 1 || go.stride(0) < width) go = go.contiguous();
    const int64_t esz = go.element_size();
    char* gbase = static_cast<char*>(go.data_ptr());
    Tensor dz, dC;
    if (need_dz) dz = at::empty({p.N, p.h}, z.options().requires_grad(false));
    if (need_dC) dC = at::empty({p.h, p.L, p.r}, z.options().requires_grad(false));
    const size_t need = skv_scratch_bytes(&p, SKV_OP_BACKWARD);
    Tensor scratch = scratch_for(need, z);
    const bool f32 = p.dtype == SKV_F32;
    const int code = skv_feature_backward(
        &p, z.data_ptr(), z.stride(0), table.data_ptr(), with_base ? gbase : nullptr, go.stride(0),
        gbase + (with_base ? p.h * esz : 0), go.stride(0), need_dz ? dz.data_ptr() : nullptr, p.h,
        need_dC && f32 ? static_cast<float*>(dC.data_ptr()) : nullptr, need_dC && !f32 ? dC.data_ptr() : nullptr,
        need ? scratch.data_ptr() : nullptr, need,
        static_cast<int32_t*>(status_word(z.device().index()).data_ptr()),
        c10::cuda::getCurrentCUDAStream(z.device().index()).stream());
    if (code) fail(code);
    out[0] = dz;
    // During graph capture dC is added into a preallocated C.grad as part of the captured work, as the
    // reference does (src/sparsespline_ffn/kernels/flash_spline_feature_autograd.py:154-172).
    if (need_dC && C.is_leaf() && C.grad().defined() &&
        c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None)
      C.mutable_grad().add_(dC);
    else
      out[1] = dC;
    return out;
  }
};

Tensor differentiable_forward(const Tensor& z, const Tensor& C, const skv_problem& p, long bwd_impl, bool with_base) {
  Tensor f = forward(z, C, p, with_base);
  if (f.defined() && at::GradMode::is_enabled() && (z.requires_grad() || C.requires_grad())) {
    auto node = std::shared_ptr<SplineFeatureBackward>(new SplineFeatureBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(z, C));
    node->z_ = torch::autograd::SavedVariable(z, false);
    node->C_ = torch::autograd::SavedVariable(C, false);
    node->p = p;
    node->p.impl = (int32_t)bwd_impl;
    node->with_base = with_base;
    torch::autograd::set_history(f, node);
  }
  return f;
}

// ------------------------------------------------------------------------------------------ Python entries
bool env_override() {
  const char* e = std::getenv("SPARSE_SPLINE_FWD_KERNEL");
  return e && *e;
}

PyObject* none() { Py_RETURN_NONE; }

bool numbers(PyObject* const* a, double* d, int n) {
  for (int i = 0; i < n; ++i) {
    d[i] = PyFloat_AsDouble(a[i]);
    if (d[i] == -1.0 && PyErr_Occurred()) { PyErr_Clear(); return false; }
  }
  return true;
}
bool integers(PyObject* const* a, long* v, int n) {
  for (int i = 0; i < n; ++i) {
    v[i] = PyLong_AsLong(a[i]);
    if (v[i] == -1 && PyErr_Occurred()) { PyErr_Clear(); return false; }
  }
  return true;
}

// (z, C, grid_lo, grid_hi, lambda, G, activation, fwd_impl, bwd_impl, spline_order, with_base) -> Tensor or None
PyObject* py_feature(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 11 || !THPVariable_Check(a[0]) || !THPVariable_Check(a[1])) return none();
  double d[3];
  long v[6];
  if (!numbers(a + 2, d, 3) || !integers(a + 5, v, 6) || env_override()) return none();
  try {
    const Tensor& z = THPVariable_Unpack(a[0]);
    const Tensor& C = THPVariable_Unpack(a[1]);
    skv_problem p;
    if (!plain_problem(z, C, d[0], d[1], v[0], v[1], d[2], v[2], v[4], &p)) return none();
    Tensor f = differentiable_forward(z, C, p, v[3], v[5] != 0);
    return f.defined() ? THPVariable_Wrap(f) : none();
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

// (z, C, W_out, grid_lo, grid_hi, lambda, G, activation) -> Tensor or None
PyObject* py_readout(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 8 || !THPVariable_Check(a[0]) || !THPVariable_Check(a[1]) || !THPVariable_Check(a[2])) return none();
  double d[3];
  long v[2];
  if (!numbers(a + 3, d, 3) || !integers(a + 6, v, 2)) return none();
  try {
    const Tensor& z = THPVariable_Unpack(a[0]);
    const Tensor& C = THPVariable_Unpack(a[1]);
    const Tensor& W = THPVariable_Unpack(a[2]);
    skv_problem p;
    if (!plain_problem(z, C, d[0], d[1], v[0], v[1], d[2], SKV_IMPL_AUTO, 2, &p) || p.dtype != SKV_BF16) return none();
    if (!z.is_contiguous() || !W.is_cuda() || W.device() != z.device() || W.scalar_type() != at::kBFloat16 ||
        W.unsafeGetTensorImpl()->is_python_dispatch() || W.dim() != 2 || !W.is_contiguous() ||
        W.size(1) != (int64_t)p.h + p.r)
      return none();
    const int64_t D = W.size(0);
    const size_t need = skv_readout_scratch_bytes(&p, D);
    if (need == 0) return none();
    c10::cuda::CUDAGuard guard(z.device());
    Tensor y = at::empty({p.N, D}, z.options().requires_grad(false));
    Tensor scratch = scratch_for(need, z);
    const int code = skv_feature_readout_forward(
        &p, z.data_ptr(), z.stride(0), C.data_ptr(), W.data_ptr(), W.stride(0), D, y.data_ptr(), y.stride(0),
        scratch.data_ptr(), need, static_cast<int32_t*>(status_word(z.device().index()).data_ptr()),
        c10::cuda::getCurrentCUDAStream(z.device().index()).stream());
    if (code) fail(code);
    return THPVariable_Wrap(y);
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

// (device index) -> the device's status word
PyObject* py_status_word(PyObject*, PyObject* arg) {
  const long dev = PyLong_AsLong(arg);
  if (dev == -1 && PyErr_Occurred()) return nullptr;
  try {
    return THPVariable_Wrap(status_word((int)dev));
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

PyMethodDef methods[] = {
    {"feature", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_feature)), METH_FASTCALL,
     "feature(z, C, grid_lo, grid_hi, lambda, G, activation, fwd_impl, bwd_impl, spline_order, with_base)"},
    {"readout", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_readout)), METH_FASTCALL,
     "readout(z, C, W_out, grid_lo, grid_hi, lambda, G, activation)"},
    {"status_word", py_status_word, METH_O, "status_word(device_index)"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "Native host path of the operators.", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) { return PyModule_Create(&module); }
