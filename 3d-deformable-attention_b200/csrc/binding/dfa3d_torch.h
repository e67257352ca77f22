// What the two halves of the native host path share: the C ABI's entry points, argument checks and small helpers
// (dfa3d_torch.cpp: the operator; dfa3d_torch_layers.cpp: the layer around it).
#pragma once
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/utils/pybind.h>

#include <ATen/ATen.h>
#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>

#include <atomic>
#include <optional>

#include "dfa3d_b200.h"

namespace dfa3d_torch {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// ------------------------------------------------------------------------------------------------
// the C ABI
// ------------------------------------------------------------------------------------------------
#define DFA3D_ENTRIES(X)                                                                                 \
  X(dfa3d_last_error) X(dfa3d_depth_score_forward) X(dfa3d_depth_score_backward)                         \
  X(dfa3d_wms_attn_forward) X(dfa3d_wms_attn_backward) X(dfa3d_fused_forward) X(dfa3d_fused_backward)    \
  X(dfa3d_msda_forward) X(dfa3d_msda_backward) X(dfa3d_attn3d_forward_rows) X(dfa3d_attn3d_backward_rows) \
  X(dfa3d_fused_forward_ragged) X(dfa3d_fused_backward_ragged) \
  X(dfa3d_dist_from_logits) X(dfa3d_dist_from_logits_backward_typed)           \
  X(dfa3d_zero_two) X(dfa3d_convert_two) X(dfa3d_attn2d_supported) X(dfa3d_attn2d_forward) X(dfa3d_attn2d_backward)           \
  X(dfa3d_rebatch_gather) X(dfa3d_rebatch_combine) X(dfa3d_add_layer_norm_forward)                       \
  X(dfa3d_add_layer_norm_infer) X(dfa3d_layer_norm_backward) X(dfa3d_column_sum)                         \
  X(dfa3d_relu_backward_column_sum) X(dfa3d_slice_sum) X(dfa3d_copy_segments)

struct Abi {
#define X(name) decltype(&::name) name = nullptr;
  DFA3D_ENTRIES(X)
#undef X
};
inline Abi lib;

inline bool bound = false;
inline std::atomic<long long> calls{0};      // successful entry-point calls

inline void check(int rc, const char *what) {
  if (rc == DFA3D_OK) {
    calls.fetch_add(1, std::memory_order_relaxed);
    return;
  }
  const char *kind = rc == DFA3D_ERR_INVALID_ARGUMENT ? "invalid argument"
                     : rc == DFA3D_ERR_UNSUPPORTED    ? "unsupported"
                                                      : "CUDA error";
  TORCH_CHECK(false, what, " failed (", kind, "): ", lib.dfa3d_last_error());
}

inline void *stream_of(const Tensor &t) { return at::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// ------------------------------------------------------------------------------------------------
// arguments
// ------------------------------------------------------------------------------------------------
// Modes in which the Python Function does something of its own.  (Under jit.trace it becomes an operation of the graph; of a
// call made here the tracer would see the allocation of the result and not the kernel that fills it.)
inline bool plain_mode() {
  return bound && !torch::jit::tracer::isTracing() && !at::autocast::is_autocast_enabled(at::kCUDA) &&
         !c10::impl::TorchDispatchModeTLS::any_modes_set() &&
         !c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode);
}

inline bool storage_type(at::ScalarType t) { return t == at::kFloat || t == at::kBFloat16 || t == at::kHalf; }

inline int dtype_code(const Tensor &t) {
  return t.scalar_type() == at::kHalf ? DFA3D_DTYPE_F16 : t.scalar_type() == at::kBFloat16 ? DFA3D_DTYPE_BF16 : DFA3D_DTYPE_F32;
}

// A plain contiguous CUDA tensor without forward-mode tangent.
inline bool plain_tensor(PyObject *o, Tensor &t) {
  if (!THPVariable_Check(o)) return false;
  t = THPVariable_Unpack(o);
  return t.is_cuda() && t.layout() == at::kStrided && t.is_contiguous() && !t.unsafeGetTensorImpl()->is_python_dispatch() &&
         !t._fw_grad(0).defined();
}

inline bool float_tensor(PyObject *o, Tensor &t, int64_t dim) {
  return plain_tensor(o, t) && t.scalar_type() == at::kFloat && (dim < 0 || t.dim() == dim);
}

inline bool long_tensor(PyObject *o, Tensor &t, int64_t dim) {
  return plain_tensor(o, t) && t.scalar_type() == at::kLong && t.dim() == dim;
}

inline bool integer(PyObject *o, int64_t &v) {
  if (!PyLong_CheckExact(o)) return false;
  v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  return true;
}

// None, or a pair of positive integers
inline bool map_argument(PyObject *o, int64_t &h, int64_t &w) {
  h = w = 0;
  if (o == Py_None) return true;
  return PyTuple_CheckExact(o) && PyTuple_GET_SIZE(o) == 2 && integer(PyTuple_GET_ITEM(o, 0), h) &&
         integer(PyTuple_GET_ITEM(o, 1), w) && h > 0 && w > 0 && h < (1 << 24) && w < (1 << 24);
}

// `batch % min(batch, im2col_step)`, as the reference demands
inline bool step_divides(PyObject *o, int64_t batch) {
  int64_t step;
  if (!integer(o, step) || step <= 0) return false;
  return batch == 0 || batch % std::min(batch, step) == 0;
}

inline bool small(const Tensor &t) {      // every size fits the descriptor's int32 fields
  for (int64_t s : t.sizes())
    if (s >= (int64_t(1) << 31)) return false;
  return true;
}

template <typename... T>
bool one_device(const Tensor &a, const T &...more) {
  return ((more.device() == a.device()) && ...);
}

inline bool sizes_are(const Tensor &t, std::initializer_list<int64_t> s) { return t.sizes() == at::IntArrayRef(s); }

// value (B,N,H,C) and dist (B,Nd,H,D) | (B,Nd,D): fills the descriptor's fields that follow from them.
inline bool describe_dist(const Tensor &dist, int64_t B, int64_t N, int64_t H, int64_t mh, int64_t mw, dfa3d_problem &p) {
  if (dist.dim() != 3 && dist.dim() != 4) return false;
  if (dist.dim() == 4 && dist.size(2) != H) return false;
  const int64_t D = dist.size(-1);
  if (dist.size(0) != B || dist.size(1) != (mh ? mh * mw : N)) return false;
  p.D = (int32_t)D;
  p.dist_dtype = dtype_code(dist);
  p.dist_head_stride = dist.dim() == 4 ? D : 0;
  p.dist_map_h = (int32_t)mh;
  p.dist_map_w = (int32_t)mw;
  return true;
}

inline void describe_value(const Tensor &value, dfa3d_problem &p) {
  p.B = (int32_t)value.size(0); p.N = (int32_t)value.size(1);
  p.H = (int32_t)value.size(2); p.C = (int32_t)value.size(3);
  p.value_dtype = dtype_code(value);
}

inline Tensor empty_f32(at::IntArrayRef sizes, const Tensor &like) {
  return at::empty(sizes, like.options().dtype(at::kFloat));
}

// Two zeroed float32 gradients (the second may be undefined), one launch for both.
inline void zero_two(const Tensor &a, const Tensor &b, void *s) {
  check(lib.dfa3d_zero_two(a.data_ptr<float>(), a.numel(), b.defined() ? b.data_ptr<float>() : nullptr,
                           b.defined() ? b.numel() : 0, s),
        "dfa3d_zero_two");
  calls.fetch_sub(1, std::memory_order_relaxed);
}

inline const float *fp(const Tensor &t) { return static_cast<const float *>(t.const_data_ptr()); }
inline float *fpm(const Tensor &t) { return static_cast<float *>(t.mutable_data_ptr()); }
inline const int64_t *lp(const Tensor &t) { return static_cast<const int64_t *>(t.const_data_ptr()); }
inline const int32_t *ip(const Tensor &t) { return static_cast<const int32_t *>(t.const_data_ptr()); }

inline bool aligned(const Tensor &t, uintptr_t bytes) { return reinterpret_cast<uintptr_t>(t.const_data_ptr()) % bytes == 0; }

// float32 and contiguous, whatever the consumer of the result handed back
inline Tensor f32(const Tensor &g) {
  if (g.scalar_type() == at::kFloat) return g.contiguous();
  if ((g.scalar_type() != at::kHalf && g.scalar_type() != at::kBFloat16) || !g.is_cuda() || !g.is_contiguous() || !aligned(g, 16))
    return g.to(at::kFloat).contiguous();
  c10::cuda::CUDAGuard guard(g.device());
  Tensor w = empty_f32(g.sizes(), g);
  check(lib.dfa3d_convert_two(dtype_code(g), 1, const_cast<void *>(g.const_data_ptr()), w.mutable_data_ptr(), g.numel(), nullptr,
                              nullptr, 0, stream_of(g)),
        "dfa3d_convert_two");
  return w;
}

// fp32 results in the types that the caller gets them in (kFloat: as they are), both 16-bit ones with one launch; undefined
// tensors stay so.
inline void narrow_two(Tensor &a, at::ScalarType ta, Tensor &b, at::ScalarType tb) {
  const bool na = a.defined() && ta != at::kFloat, nb = b.defined() && tb != at::kFloat;
  if (!na && !nb) return;
  if (na && nb && ta != tb) {
    a = a.to(ta);
    b = b.to(tb);
    return;
  }
  c10::cuda::CUDAGuard guard((na ? a : b).device());
  Tensor ra, rb;
  if (na) ra = at::empty(a.sizes(), a.options().dtype(ta));
  if (nb) rb = at::empty(b.sizes(), b.options().dtype(tb));
  check(lib.dfa3d_convert_two(dtype_code(na ? ra : rb), 0, na ? ra.mutable_data_ptr() : nullptr,
                              na ? a.mutable_data_ptr() : nullptr, na ? a.numel() : 0, nb ? rb.mutable_data_ptr() : nullptr,
                              nb ? b.mutable_data_ptr() : nullptr, nb ? b.numel() : 0, stream_of(na ? a : b)),
        "dfa3d_convert_two");
  if (na) a = ra;
  if (nb) b = rb;
}

// What a node keeps from its forward: the tensors, which pass through the saved-tensor hooks in force, and beside them what
// they were.  The kernels read them by address, so what a hook hands back has to be of the same type, size and device; its
// layout may be another.
struct Kept : torch::CustomClassHolder {
  struct Was {
    int64_t numel;
    at::ScalarType type;
    c10::Device device;
  };
  c10::SmallVector<Was, 9> was;
};

template <typename X>
void keep(AutogradContext *ctx, const c10::intrusive_ptr<X> &x, variable_list tensors) {
  for (const Tensor &t : tensors) {
    if (t.defined()) x->was.push_back({t.numel(), t.scalar_type(), t.device()});
    else x->was.push_back({-1, at::kFloat, at::kCPU});
  }
  ctx->save_for_backward(std::move(tensors));
  ctx->saved_data["x"] = c10::IValue::make_capsule(x);
}

template <typename X>
c10::intrusive_ptr<X> kept(AutogradContext *ctx, variable_list &tensors) {
  const auto x = c10::static_intrusive_pointer_cast<X>(ctx->saved_data.at("x").toCapsule());
  tensors = ctx->get_saved_variables();
  TORCH_CHECK(tensors.size() == x->was.size(), "saved tensors are missing");
  for (size_t i = 0; i < tensors.size(); ++i) {
    Tensor &t = tensors[i];
    const Kept::Was &w = x->was[i];
    TORCH_CHECK(t.defined() ? t.numel() == w.numel && t.scalar_type() == w.type && t.device() == w.device : w.numel < 0,
                "a saved-tensor hook returned a tensor of another type, size or device than it was given");
    if (t.defined()) t = t.contiguous();
  }
  return x;
}

// Gradients of a backward that must not be differentiated again: with create_graph the results get a node that
// says so when it is reached (torch.autograd.function.once_differentiable does the same).
inline variable_list once(variable_list out, const variable_list &grads) {
  if (!at::GradMode::is_enabled()) return out;
  bool any = false;
  for (const auto &g : grads) any |= g.defined() && g.requires_grad();
  if (!any) return out;
  std::vector<size_t> where;
  variable_list in;
  for (size_t i = 0; i < out.size(); ++i)
    if (out[i].defined()) {
      where.push_back(i);
      in.push_back(out[i].detach().requires_grad_(true));
    }
  auto err = std::make_shared<torch::autograd::DelayedError>(
      "trying to differentiate twice a function that was marked with @once_differentiable", (int64_t)in.size());
  auto res = (*err)(std::move(in));
  for (size_t i = 0; i < where.size(); ++i) out[where[i]] = res[i];
  return out;
}

// A gradient that flows into the returned depth_score is not supported (as in the reference): zero is tolerated.
inline void refuse_score_gradient(const Tensor &g) {
  TORCH_CHECK_NOT_IMPLEMENTED(!g.defined() || g.sum().item<double>() == 0.0,
                              "no gradient can flow into the returned depth_score");
}

template <typename... T>
bool wants_grad(const T &...t) {
  return at::GradMode::is_enabled() && (t.requires_grad() || ...);
}

// torch::autograd::Function takes tensors that may be absent as optionals
inline std::optional<Tensor> given(const Tensor &t) { return t.defined() ? std::optional<Tensor>(t) : std::nullopt; }

inline PyObject *not_plain() { Py_RETURN_NOTIMPLEMENTED; }

// A weight gradient of at least so many rows is formed as so many slices of them (dfa3d_torch_layers.cpp; the Python
// Function does the same, layer_ops.py)
constexpr int64_t kSplitRows = 16384, kSplits = 16;

extern PyMethodDef layer_methods[];      // dfa3d_torch_layers.cpp, ends in a null entry

}  // namespace dfa3d_torch
