// Native host path of the autograd Functions: argument checks, output allocation, the kernel call and the
// autograd node in C++, so that a small call is not bound by the interpreter.
//
// What a call costs on the host decides every problem below a few hundred microseconds of kernels: a forward +
// backward of the one-stage operator on 512 queries spent 190 us in Python (argument checks, ctypes, the
// Function machinery twice) around 34 us of kernels; here the same pass is a handful of microseconds a side.
//
// Every function takes exactly the positional arguments of the Python Function's forward and returns either its
// result or NotImplemented.  NotImplemented means "not the plain case": a dtype, layout, size or mode that is not
// handled here (double precision, autocast, functorch, forward-mode AD, tracing, anything inconsistent).  The
// caller then runs the Python Function, which covers everything and raises the documented errors; so no check is
// written twice with two different messages.
//
// Kernels are reached through the C ABI (include/dfa3d_b200.h) of the library the Python side has loaded:
// bind() receives the entry points' addresses.
#include "dfa3d_torch.h"

using namespace dfa3d_torch;

namespace {

// ------------------------------------------------------------------------------------------------
// autograd nodes; what they keep beside their tensors travels with them in one capsule
// ------------------------------------------------------------------------------------------------
struct Extra : Kept {
  dfa3d_problem p;
  int64_t Z = 0;
  bool half = false;
};

// ---- one-stage operator, dense and ragged ----------------------------------------------------------
// Result tensors of the forward: out and, when asked for, the depth scores.
variable_list fused_forward(const dfa3d_problem &p, const Tensor &value, const Tensor &dist, const Tensor &shapes,
                            const Tensor &lsi, const Tensor &loc, const Tensor &attn, const Tensor &q_off,
                            bool need_score) {
  c10::cuda::CUDAGuard guard(value.device());
  std::vector<int64_t> lead(loc.sizes().begin(), loc.sizes().end());
  const bool ragged = q_off.defined();
  Tensor out = ragged ? empty_f32({loc.size(0), (int64_t)p.H * p.C}, value)
                      : empty_f32({loc.size(0), loc.size(1), (int64_t)p.H * p.C}, value);
  Tensor score;
  if (need_score) {
    lead.back() = 4;
    score = empty_f32(lead, value);
  }
  void *s = stream_of(value);
  float *ds = need_score ? fpm(score) : nullptr;
  if (ragged)
    check(lib.dfa3d_fused_forward_ragged(&p, ip(q_off), value.const_data_ptr(), dist.const_data_ptr(), lp(shapes),
                                         lp(lsi), fp(loc), fp(attn), fpm(out), ds, s),
          "dfa3d_fused_forward_ragged");
  else
    check(lib.dfa3d_fused_forward(&p, value.const_data_ptr(), dist.const_data_ptr(), lp(shapes), lp(lsi), fp(loc),
                                  fp(attn), fpm(out), ds, s),
          "dfa3d_fused_forward");
  return {out, score};
}

struct FusedFn : torch::autograd::Function<FusedFn> {
  static variable_list forward(AutogradContext *ctx, const Tensor &value, const Tensor &dist, const Tensor &shapes,
                               const Tensor &lsi, const Tensor &loc, const Tensor &attn,
                               const std::optional<Tensor> &offsets, bool need_score, c10::intrusive_ptr<Extra> x) {
    ctx->set_materialize_grads(false);
    const Tensor q_off = offsets.value_or(Tensor());
    auto out = fused_forward(x->p, value, dist, shapes, lsi, loc, attn, q_off, need_score);
    if (x->half) narrow_two(out[0], at::kHalf, out[1], at::kHalf);
    keep(ctx, x, {value, dist, shapes, lsi, loc, attn, q_off});
    if (!need_score) out.pop_back();
    return out;
  }
  static variable_list backward(AutogradContext *ctx, variable_list grads) {
    variable_list none(9);
    if (grads.size() > 1) refuse_score_gradient(grads[1]);
    if (!grads[0].defined()) return none;
    variable_list v;
    const auto x = kept<Extra>(ctx, v);
    const Tensor &value = v[0], &dist = v[1], &loc = v[4], &attn = v[5], &q_off = v[6];
    c10::cuda::CUDAGuard guard(value.device());
    const Tensor go = f32(grads[0]);
    Tensor gv = empty_f32(value.sizes(), value), gd = empty_f32(dist.sizes(), dist);
    Tensor gl = at::empty_like(loc), ga = at::empty_like(attn);
    void *s = stream_of(value);
    zero_two(gv, gd, s);
    if (q_off.defined())
      check(lib.dfa3d_fused_backward_ragged(&x->p, ip(q_off), value.const_data_ptr(), dist.const_data_ptr(), lp(v[2]),
                                            lp(v[3]), fp(loc), fp(attn), fp(go), fpm(gv), fpm(gd), fpm(gl), fpm(ga), s),
            "dfa3d_fused_backward_ragged");
    else
      check(lib.dfa3d_fused_backward(&x->p, value.const_data_ptr(), dist.const_data_ptr(), lp(v[2]), lp(v[3]), fp(loc),
                                     fp(attn), fp(go), fpm(gv), fpm(gd), fpm(gl), fpm(ga), s),
            "dfa3d_fused_backward");
    // what autograd would convert after this node
    narrow_two(gv, ctx->needs_input_grad(0) ? value.scalar_type() : at::kFloat, gd,
               ctx->needs_input_grad(1) ? dist.scalar_type() : at::kFloat);
    return once({gv, gd, Tensor(), Tensor(), gl, ga, Tensor(), Tensor(), Tensor()}, grads);
  }
};

// ---- operator fed with offsets and logits, dense and ragged ------------------------------------------
Tensor attn3d_forward(const Extra &x, const Tensor &value, const Tensor &dist, const Tensor &shapes, const Tensor &lsi,
                      const Tensor &ref, const Tensor &uv, const Tensor &od, const Tensor &logits,
                      const Tensor &q_off) {
  c10::cuda::CUDAGuard guard(value.device());
  const dfa3d_problem &p = x.p;
  const bool ragged = q_off.defined();
  Tensor out = ragged ? empty_f32({uv.size(0), (int64_t)p.H * p.C}, value)
                      : empty_f32({uv.size(0), uv.size(1), (int64_t)p.H * p.C}, value);
  void *s = stream_of(value);
  check(lib.dfa3d_attn3d_forward_rows(&p, (int32_t)x.Z, (int32_t)shapes.size(1), 0, 0, ragged ? ip(q_off) : nullptr, nullptr,
                                        value.const_data_ptr(), dist.const_data_ptr(), lp(shapes), lp(lsi), fp(ref), fp(uv),
                                        fp(od), fp(logits), fpm(out), s),
        "dfa3d_attn3d_forward");
  return out;
}

struct Attn3dFn : torch::autograd::Function<Attn3dFn> {
  static Tensor forward(AutogradContext *ctx, const Tensor &value, const Tensor &dist, const Tensor &shapes,
                        const Tensor &lsi, const Tensor &ref, const Tensor &uv, const Tensor &od,
                        const Tensor &logits, const std::optional<Tensor> &offsets,
                        c10::intrusive_ptr<Extra> x) {
    const Tensor q_off = offsets.value_or(Tensor());
    Tensor out = attn3d_forward(*x, value, dist, shapes, lsi, ref, uv, od, logits, q_off);
    keep(ctx, x, {value, dist, shapes, lsi, ref, uv, od, logits, q_off});
    return out;
  }
  static variable_list backward(AutogradContext *ctx, variable_list grads) {
    variable_list v;
    const auto x = kept<Extra>(ctx, v);
    const Tensor &value = v[0], &dist = v[1], &uv = v[5], &od = v[6], &logits = v[7], &q_off = v[8];
    c10::cuda::CUDAGuard guard(value.device());
    const Tensor go = f32(grads[0]);
    Tensor gv = empty_f32(value.sizes(), value), gd = empty_f32(dist.sizes(), dist);
    Tensor guv = at::empty_like(uv), god = at::empty_like(od), gl = at::empty_like(logits);
    void *s = stream_of(value);
    zero_two(gv, gd, s);
    check(lib.dfa3d_attn3d_backward_rows(&x->p, (int32_t)x->Z, (int32_t)v[2].size(1), 0, 0, q_off.defined() ? ip(q_off) : nullptr,
                                           value.const_data_ptr(), dist.const_data_ptr(), lp(v[2]), lp(v[3]), fp(v[4]),
                                           fp(uv), fp(od), fp(logits), fp(go), fpm(gv), fpm(gd), fpm(guv), fpm(god), fpm(gl),
                                           s),
          "dfa3d_attn3d_backward");
    return once({gv, gd, Tensor(), Tensor(), Tensor(), guv, god, gl, Tensor(), Tensor()}, grads);
  }
};

// ---- the same with offsets, depth offsets and logits side by side in one row per query --------------------
Tensor attn3d_joint_forward(const Extra &x, const Tensor &value, const Tensor &dist, const Tensor &shapes, const Tensor &lsi,
                            const Tensor &ref, const Tensor &joint, const Tensor &q_off, const Tensor &q_row) {
  c10::cuda::CUDAGuard guard(value.device());
  std::vector<int64_t> sz(joint.sizes().begin(), joint.sizes().end());
  const int64_t row = sz.back(), part = row / 4;
  sz.front() = ref.size(0);
  sz.back() = (int64_t)x.p.H * x.p.C;
  Tensor out = empty_f32(sz, value);
  check(lib.dfa3d_attn3d_forward_rows(&x.p, (int32_t)x.Z, (int32_t)shapes.size(1), row, row,
                                      q_off.defined() ? ip(q_off) : nullptr, q_row.defined() ? ip(q_row) : nullptr,
                                      value.const_data_ptr(), dist.const_data_ptr(), lp(shapes), lp(lsi), fp(ref), fp(joint),
                                      fp(joint) + 2 * part, fp(joint) + 3 * part, fpm(out), stream_of(value)),
        "dfa3d_attn3d_forward");
  return out;
}

struct Attn3dJointFn : torch::autograd::Function<Attn3dJointFn> {
  static Tensor forward(AutogradContext *ctx, const Tensor &value, const Tensor &dist, const Tensor &shapes,
                        const Tensor &lsi, const Tensor &ref, const Tensor &joint, const std::optional<Tensor> &offsets,
                        c10::intrusive_ptr<Extra> x) {
    const Tensor q_off = offsets.value_or(Tensor());
    keep(ctx, x, {value, dist, shapes, lsi, ref, joint, q_off});
    return attn3d_joint_forward(*x, value, dist, shapes, lsi, ref, joint, q_off, Tensor());
  }
  static variable_list backward(AutogradContext *ctx, variable_list grads) {
    variable_list v;
    const auto x = kept<Extra>(ctx, v);
    const Tensor &value = v[0], &dist = v[1], &joint = v[5], &q_off = v[6];
    c10::cuda::CUDAGuard guard(value.device());
    const Tensor go = f32(grads[0]);
    Tensor gv = empty_f32(value.sizes(), value), gd = empty_f32(dist.sizes(), dist), gj = at::empty_like(joint);
    const int64_t row = joint.size(-1), part = row / 4;
    void *s = stream_of(value);
    zero_two(gv, gd, s);
    check(lib.dfa3d_attn3d_backward_rows(&x->p, (int32_t)x->Z, (int32_t)v[2].size(1), row, row,
                                         q_off.defined() ? ip(q_off) : nullptr, value.const_data_ptr(), dist.const_data_ptr(),
                                         lp(v[2]), lp(v[3]), fp(v[4]), fp(joint), fp(joint) + 2 * part, fp(joint) + 3 * part,
                                         fp(go), fpm(gv), fpm(gd), fpm(gj), fpm(gj) + 2 * part, fpm(gj) + 3 * part, s),
          "dfa3d_attn3d_backward");
    return once({gv, gd, Tensor(), Tensor(), Tensor(), gj, Tensor(), Tensor()}, grads);
  }
};

// ---- 2-D attention: with given depth scores, or plain (score undefined) --------------------------------
Tensor attn2d_forward(const dfa3d_problem &p, const Tensor &value, const Tensor &shapes, const Tensor &lsi,
                      const Tensor &loc, const Tensor &attn, const Tensor &score) {
  c10::cuda::CUDAGuard guard(value.device());
  Tensor out = empty_f32({loc.size(0), loc.size(1), (int64_t)p.H * p.C}, value);
  void *s = stream_of(value);
  if (score.defined())
    check(lib.dfa3d_wms_attn_forward(&p, value.const_data_ptr(), lp(shapes), lp(lsi), fp(loc), fp(attn), fp(score),
                                     fpm(out), s),
          "dfa3d_wms_attn_forward");
  else
    check(lib.dfa3d_msda_forward(&p, value.const_data_ptr(), lp(shapes), lp(lsi), fp(loc), fp(attn), fpm(out), s),
          "dfa3d_msda_forward");
  return out;
}

struct Attn2dFn : torch::autograd::Function<Attn2dFn> {
  static Tensor forward(AutogradContext *ctx, const Tensor &value, const Tensor &shapes, const Tensor &lsi,
                        const Tensor &loc, const Tensor &attn, const std::optional<Tensor> &scores,
                        c10::intrusive_ptr<Extra> x) {
    const Tensor score = scores.value_or(Tensor());
    Tensor out = attn2d_forward(x->p, value, shapes, lsi, loc, attn, score);
    if (x->half) out = out.to(at::kHalf);
    keep(ctx, x, {value, shapes, lsi, loc, attn, score});
    return out;
  }
  static variable_list backward(AutogradContext *ctx, variable_list grads) {
    variable_list v;
    const auto x = kept<Extra>(ctx, v);
    const Tensor &value = v[0], &loc = v[3], &attn = v[4], &score = v[5];
    c10::cuda::CUDAGuard guard(value.device());
    const Tensor go = f32(grads[0]);
    Tensor gv = empty_f32(value.sizes(), value), gl = at::empty_like(loc), ga = at::empty_like(attn), gs;
    void *s = stream_of(value);
    zero_two(gv, Tensor(), s);
    if (score.defined()) {
      gs = at::empty_like(score);
      check(lib.dfa3d_wms_attn_backward(&x->p, value.const_data_ptr(), lp(v[1]), lp(v[2]), fp(loc), fp(attn), fp(score),
                                        fp(go), fpm(gv), fpm(gl), fpm(ga), fpm(gs), s),
            "dfa3d_wms_attn_backward");
    } else {
      check(lib.dfa3d_msda_backward(&x->p, value.const_data_ptr(), lp(v[1]), lp(v[2]), fp(loc), fp(attn), fp(go),
                                    fpm(gv), fpm(gl), fpm(ga), s),
            "dfa3d_msda_backward");
    }
    return once({gv, Tensor(), Tensor(), gl, ga, gs, Tensor()}, grads);
  }
};

// ---- depth scores alone -----------------------------------------------------------------------------
Tensor depth_score_forward(const dfa3d_problem &p, const Tensor &dist, const Tensor &shapes, const Tensor &lsi,
                           const Tensor &loc) {
  c10::cuda::CUDAGuard guard(dist.device());
  std::vector<int64_t> sz(loc.sizes().begin(), loc.sizes().end());
  sz.back() = 4;
  Tensor out = empty_f32(sz, dist);
  check(lib.dfa3d_depth_score_forward(&p, dist.const_data_ptr(), lp(shapes), lp(lsi), fp(loc), fpm(out),
                                      stream_of(dist)),
        "dfa3d_depth_score_forward");
  return out;
}

struct DepthScoreFn : torch::autograd::Function<DepthScoreFn> {
  static Tensor forward(AutogradContext *ctx, const Tensor &dist, const Tensor &shapes, const Tensor &lsi,
                        const Tensor &loc, c10::intrusive_ptr<Extra> x) {
    Tensor out = depth_score_forward(x->p, dist, shapes, lsi, loc);
    keep(ctx, x, {dist, shapes, lsi, loc});
    return out;
  }
  static variable_list backward(AutogradContext *ctx, variable_list grads) {
    variable_list v;
    const auto x = kept<Extra>(ctx, v);
    const Tensor &dist = v[0], &loc = v[3];
    c10::cuda::CUDAGuard guard(dist.device());
    const Tensor go = f32(grads[0]);
    Tensor gd = empty_f32(dist.sizes(), dist), gl = at::empty_like(loc);
    void *s = stream_of(dist);
    zero_two(gd, Tensor(), s);
    check(lib.dfa3d_depth_score_backward(&x->p, dist.const_data_ptr(), lp(v[1]), lp(v[2]), fp(loc), fp(go), fpm(gd),
                                         fpm(gl), s),
          "dfa3d_depth_score_backward");
    return once({gd, Tensor(), Tensor(), gl, Tensor()}, grads);
  }
};

// ---- depth distribution from logits -------------------------------------------------------------------
struct DistArgs : Kept {
  int32_t N = 0, act = 0, dtype = 0;
};

Tensor dist_forward(const DistArgs &a, const Tensor &logits, const Tensor &shapes, const Tensor &lsi,
                    at::ScalarType type) {
  c10::cuda::CUDAGuard guard(logits.device());
  const int32_t B = (int32_t)logits.size(0), D = (int32_t)logits.size(1);
  Tensor dist = at::empty({B, a.N, D}, logits.options().dtype(type));
  check(lib.dfa3d_dist_from_logits(fp(logits), B, D, (int32_t)logits.size(2), (int32_t)logits.size(3), lp(shapes),
                                   (int32_t)shapes.size(1), lp(lsi), (int32_t)shapes.size(0), a.N, a.act, a.dtype,
                                   dist.mutable_data_ptr(), stream_of(logits)),
        "dfa3d_dist_from_logits");
  return dist;
}

struct DistFn : torch::autograd::Function<DistFn> {
  static Tensor forward(AutogradContext *ctx, const Tensor &logits, const Tensor &shapes, const Tensor &lsi,
                        c10::intrusive_ptr<DistArgs> a, int64_t type) {
    Tensor dist = dist_forward(*a, logits, shapes, lsi, static_cast<at::ScalarType>(type));
    keep(ctx, a, {logits, shapes, lsi});
    return dist;
  }
  static variable_list backward(AutogradContext *ctx, variable_list grads) {
    variable_list v;
    const auto a = kept<DistArgs>(ctx, v);
    const Tensor &logits = v[0];
    c10::cuda::CUDAGuard guard(logits.device());
    const Tensor go = storage_type(grads[0].scalar_type()) ? grads[0].contiguous() : f32(grads[0]);
    Tensor gl = at::empty_like(logits);
    check(lib.dfa3d_dist_from_logits_backward_typed(fp(logits), (int32_t)logits.size(0), (int32_t)logits.size(1),
                                              (int32_t)logits.size(2), (int32_t)logits.size(3), lp(v[1]),
                                              (int32_t)v[1].size(1), lp(v[2]), (int32_t)v[1].size(0), a->N, a->act,
                                              dtype_code(go), go.const_data_ptr(), fpm(gl), stream_of(logits)),
          "dfa3d_dist_from_logits_backward");
    return once({gl, Tensor(), Tensor(), Tensor(), Tensor()}, grads);
  }
};

// ------------------------------------------------------------------------------------------------
// Python entry points (METH_FASTCALL: no tuple, no keyword parsing)
// ------------------------------------------------------------------------------------------------
// (out, score or None)
PyObject *pair(const variable_list &r) {
  PyObject *res = PyTuple_New(2);
  if (!res) throw python_error();
  PyTuple_SET_ITEM(res, 0, THPVariable_Wrap(r[0]));
  if (r.size() > 1 && r[1].defined()) {
    PyTuple_SET_ITEM(res, 1, THPVariable_Wrap(r[1]));
  } else {
    Py_INCREF(Py_None);
    PyTuple_SET_ITEM(res, 1, Py_None);
  }
  return res;
}

// The half-storage variant: value and dist stay half, other half tensors are widened, results come back as half.
// Applies when any tensor is half; otherwise the call is the plain one.
struct Half {
  bool on = false;
  void see(PyObject *o) {
    if (THPVariable_Check(o)) on |= THPVariable_Unpack(o).scalar_type() == at::kHalf;
  }
};

PyObject *run_fused(PyObject *const *a, Py_ssize_t n, bool ragged, bool fp16) {
  // value, dist, shapes, lsi, loc, attn, (im2col_step | q_off, max_queries) [, return_depth_score [, dist_map]]
  const Py_ssize_t fixed = ragged ? 8 : 7;
  if (n < fixed || n > fixed + 2 || !plain_mode()) return not_plain();
  Half half;
  if (fp16)
    for (int i : {0, 1, 4, 5}) half.see(a[i]);
  if (half.on && (THPVariable_Check(a[4]) ? THPVariable_Unpack(a[4]).scalar_type() != at::kFloat : true)) return not_plain();
  Tensor value, dist, shapes, lsi, loc, attn, q_off;
  int64_t mh = 0, mw = 0, max_q = 0;
  if (!plain_tensor(a[0], value) || !plain_tensor(a[1], dist) || !long_tensor(a[2], shapes, 2) || !long_tensor(a[3], lsi, 1) ||
      !float_tensor(a[4], loc, ragged ? 5 : 6) || !float_tensor(a[5], attn, ragged ? 4 : 5))
    return not_plain();
  bool need_score = true;
  if (n > fixed) {
    if (!PyBool_Check(a[fixed])) return not_plain();
    need_score = a[fixed] == Py_True;
  }
  if (n > fixed + 1 && !map_argument(a[fixed + 1], mh, mw)) return not_plain();
  if (value.dim() != 4 || !storage_type(value.scalar_type()) || !storage_type(dist.scalar_type()) || !small(value) ||
      !small(dist) || !small(loc) || !one_device(value, dist, shapes, lsi, loc, attn))
    return not_plain();
  if (half.on && (value.scalar_type() != at::kHalf || dist.scalar_type() != at::kHalf)) return not_plain();
  const int64_t B = value.size(0), H = value.size(2), k = ragged ? 1 : 2;      // dimension of the heads in loc
  const int64_t L = loc.size(k + 1), P = loc.size(k + 2);
  if (loc.size(-1) != 3 || loc.size(k) != H || !sizes_are(shapes, {L, 3}) || lsi.size(0) != L ||
      attn.sizes() != loc.sizes().slice(0, k + 3))
    return not_plain();
  auto x = c10::make_intrusive<Extra>();
  dfa3d_problem &p = x->p;
  memset(&p, 0, sizeof p);
  describe_value(value, p);
  if (!describe_dist(dist, B, value.size(1), H, mh, mw, p)) return not_plain();
  if (ragged) {
    if (!plain_tensor(a[6], q_off) || q_off.scalar_type() != at::kInt || q_off.numel() != B + 1 || !one_device(value, q_off) ||
        !integer(a[7], max_q) || max_q < 0 || max_q >= (int64_t(1) << 31))
      return not_plain();
    p.Q = (int32_t)max_q;
  } else {
    if (loc.size(0) != B || !step_divides(a[6], B)) return not_plain();
    p.Q = (int32_t)loc.size(1);
  }
  p.L = (int32_t)L;
  p.P = (int32_t)P;
  x->half = half.on;
  variable_list r;
  {
    pybind11::gil_scoped_release nogil;
    if (wants_grad(value, dist, loc, attn)) {
      r = FusedFn::apply(value, dist, shapes, lsi, loc, attn, given(q_off), need_score, x);
    } else {
      r = fused_forward(p, value, dist, shapes, lsi, loc, attn, q_off, need_score);
      if (half.on) narrow_two(r[0], at::kHalf, r[1], at::kHalf);
    }
  }
  return pair(r);
}

PyObject *run_attn3d(PyObject *const *a, Py_ssize_t n, bool ragged) {
  // value, dist, shapes, lsi, ref, off_uv, off_d, logits [, q_off, max_queries] [, dist_map]
  const Py_ssize_t fixed = ragged ? 10 : 8;
  if (n < fixed || n > fixed + 1 || !plain_mode()) return not_plain();
  Tensor value, dist, shapes, lsi, ref, uv, od, logits, q_off;
  int64_t mh = 0, mw = 0, max_q = 0;
  const int64_t k = ragged ? 1 : 2;
  if (!plain_tensor(a[0], value) || !plain_tensor(a[1], dist) || !long_tensor(a[2], shapes, 2) || !long_tensor(a[3], lsi, 1) ||
      !float_tensor(a[4], ref, k + 2) || !float_tensor(a[5], uv, k + 4) || !float_tensor(a[6], od, -1) ||
      !float_tensor(a[7], logits, -1))
    return not_plain();
  if (n > fixed && !map_argument(a[fixed], mh, mw)) return not_plain();
  if (value.dim() != 4 || !storage_type(value.scalar_type()) || !storage_type(dist.scalar_type()) || !small(value) ||
      !small(dist) || !small(uv) || !one_device(value, dist, shapes, lsi, ref, uv, od, logits))
    return not_plain();
  const int64_t B = value.size(0), H = value.size(2), L = uv.size(k + 1), P = uv.size(k + 2), Z = ref.size(k);
  const int64_t pts = uv.numel() / 2;
  if (uv.size(-1) != 2 || uv.size(k) != H || ref.size(-1) != 3 || Z <= 0 || P % Z != 0 ||
      !sizes_are(shapes, {L, 3}) || lsi.size(0) != L ||
      od.numel() != pts || logits.numel() != pts || ref.size(0) != uv.size(0))
    return not_plain();
  auto x = c10::make_intrusive<Extra>();
  dfa3d_problem &p = x->p;
  memset(&p, 0, sizeof p);
  describe_value(value, p);
  if (!describe_dist(dist, B, value.size(1), H, mh, mw, p)) return not_plain();
  if (ragged) {
    if (!plain_tensor(a[8], q_off) || q_off.scalar_type() != at::kInt || q_off.numel() != B + 1 || !one_device(value, q_off) ||
        !integer(a[9], max_q) || max_q < 0 || max_q >= (int64_t(1) << 31) || od.size(0) != uv.size(0) ||
        logits.size(0) != uv.size(0))
      return not_plain();
    p.Q = (int32_t)max_q;
  } else {
    if (uv.size(0) != B || ref.size(1) != uv.size(1)) return not_plain();
    p.Q = (int32_t)uv.size(1);
  }
  p.L = (int32_t)L;
  p.P = (int32_t)P;
  x->Z = Z;
  Tensor r;
  {
    pybind11::gil_scoped_release nogil;
    r = wants_grad(value, dist, uv, od, logits)
            ? Attn3dFn::apply(value, dist, shapes, lsi, ref, uv, od, logits, given(q_off), x)
            : attn3d_forward(*x, value, dist, shapes, lsi, ref, uv, od, logits, q_off);
  }
  return THPVariable_Wrap(r);
}

PyObject *run_attn3d_joint(PyObject *const *a, Py_ssize_t n) {
  // value (B, N, H*C), dist (B, Nd, D), shapes (L, 2), lsi, ref (.., Z, 3), joint (.., 4*H*L*P), heads, points,
  // q_off or None, max_queries, dist_map, q_row or None; ".." is B, Q or, with q_off, R -- of joint, with q_row, any number
  int64_t H, P, max_q = 0, mh, mw;
  if (n != 12 || !plain_mode() || !integer(a[6], H) || !integer(a[7], P) || !map_argument(a[10], mh, mw)) return not_plain();
  const bool ragged = a[8] != Py_None;
  const int64_t k = ragged ? 1 : 2;
  Tensor value, dist, shapes, lsi, ref, joint, q_off, q_row;
  if (!plain_tensor(a[0], value) || value.dim() != 3 || !plain_tensor(a[1], dist) || dist.dim() != 3 ||
      !long_tensor(a[2], shapes, 2) || !long_tensor(a[3], lsi, 1) || !float_tensor(a[4], ref, k + 2) ||
      !float_tensor(a[5], joint, k + 1))
    return not_plain();
  if (H <= 0 || P <= 0 || value.size(2) % H != 0 || !storage_type(value.scalar_type()) || !storage_type(dist.scalar_type()) ||
      !small(value) || !small(dist) || !small(joint) || !one_device(value, dist, shapes, lsi, ref, joint) ||
      ref.requires_grad())
    return not_plain();
  const int64_t B = value.size(0), L = shapes.size(0), Z = ref.size(k);
  if (shapes.size(1) != 2 || lsi.size(0) != L || ref.size(-1) != 3 || Z <= 0 || P % Z != 0 || joint.size(-1) != 4 * H * L * P)
    return not_plain();
  auto x = c10::make_intrusive<Extra>();
  dfa3d_problem &p = x->p;
  memset(&p, 0, sizeof p);
  p.B = (int32_t)B; p.N = (int32_t)value.size(1); p.H = (int32_t)H; p.C = (int32_t)(value.size(2) / H);
  p.value_dtype = dtype_code(value);
  if (!describe_dist(dist, B, value.size(1), H, mh, mw, p)) return not_plain();
  if (ragged) {
    if (!plain_tensor(a[8], q_off) || q_off.scalar_type() != at::kInt || q_off.numel() != B + 1 || !one_device(value, q_off) ||
        !integer(a[9], max_q) || max_q < 0 || max_q >= (int64_t(1) << 31))
      return not_plain();
    p.Q = (int32_t)max_q;
    if (a[11] != Py_None) {                      // no backward
      if (!plain_tensor(a[11], q_row) || q_row.scalar_type() != at::kInt || q_row.numel() < ref.size(0) ||
          !one_device(value, q_row) || wants_grad(value, dist, joint))
        return not_plain();
    } else if (ref.size(0) != joint.size(0)) {
      return not_plain();
    }
  } else {
    if (a[11] != Py_None || ref.size(0) != B || joint.size(0) != B || ref.size(1) != joint.size(1)) return not_plain();
    p.Q = (int32_t)joint.size(1);
  }
  p.L = (int32_t)L; p.P = (int32_t)P;
  x->Z = Z;
  Tensor r;
  {
    pybind11::gil_scoped_release nogil;
    r = wants_grad(value, dist, joint) ? Attn3dJointFn::apply(value, dist, shapes, lsi, ref, joint, given(q_off), x)
                                       : attn3d_joint_forward(*x, value, dist, shapes, lsi, ref, joint, q_off, q_row);
  }
  return THPVariable_Wrap(r);
}

PyObject *run_attn2d(PyObject *const *a, Py_ssize_t n, bool scores, bool fp16) {
  // value, shapes, lsi, loc, attn [, depth_score], im2col_step
  if (n != (scores ? 7 : 6) || !plain_mode()) return not_plain();
  Half half;
  if (fp16)
    for (int i = 0; i < (scores ? 6 : 5); ++i) half.see(a[i]);
  Tensor value, shapes, lsi, loc, attn, score;
  if (!plain_tensor(a[0], value) || !long_tensor(a[1], shapes, 2) || !long_tensor(a[2], lsi, 1) || !float_tensor(a[3], loc, 6) ||
      !float_tensor(a[4], attn, 5) || (scores && !float_tensor(a[5], score, 6)))
    return not_plain();
  if (value.dim() != 4 || !storage_type(value.scalar_type()) || !small(value) || !small(loc) ||
      !one_device(value, shapes, lsi, loc, attn) || (scores && !one_device(value, score)))
    return not_plain();
  if (half.on && value.scalar_type() != at::kHalf) return not_plain();
  const int64_t B = value.size(0), H = value.size(2), Q = loc.size(1), L = loc.size(3), P = loc.size(4);
  if (loc.size(0) != B || loc.size(2) != H || loc.size(5) != 2 || !sizes_are(shapes, {L, 2}) || lsi.size(0) != L ||
      !sizes_are(attn, {B, Q, H, L, P}) || (scores && !sizes_are(score, {B, Q, H, L, P, 4})) ||
      !step_divides(a[scores ? 6 : 5], B))
    return not_plain();
  auto x = c10::make_intrusive<Extra>();
  dfa3d_problem &p = x->p;
  memset(&p, 0, sizeof p);
  describe_value(value, p);
  p.D = 1; p.L = (int32_t)L; p.Q = (int32_t)Q; p.P = (int32_t)P;
  p.dist_dtype = DFA3D_DTYPE_F32;
  x->half = half.on;
  Tensor r;
  {
    pybind11::gil_scoped_release nogil;
    if (wants_grad(value, loc, attn) || (scores && wants_grad(score))) {
      r = Attn2dFn::apply(value, shapes, lsi, loc, attn, given(score), x);
    } else {
      r = attn2d_forward(p, value, shapes, lsi, loc, attn, score);
      if (half.on) r = r.to(at::kHalf);
    }
  }
  return THPVariable_Wrap(r);
}

PyObject *run_depth_score(PyObject *const *a, Py_ssize_t n) {
  // dist, shapes, lsi, loc, im2col_step
  if (n != 5 || !plain_mode()) return not_plain();
  Tensor dist, shapes, lsi, loc;
  if (!plain_tensor(a[0], dist) || !long_tensor(a[1], shapes, 2) || !long_tensor(a[2], lsi, 1) || !float_tensor(a[3], loc, 6))
    return not_plain();
  if (!storage_type(dist.scalar_type()) || !small(dist) || !small(loc) || !one_device(dist, shapes, lsi, loc) || dist.dim() < 3)
    return not_plain();
  const int64_t B = loc.size(0), Q = loc.size(1), H = loc.size(2), L = loc.size(3), P = loc.size(4);
  if (loc.size(5) != 3 || !sizes_are(shapes, {L, 3}) || lsi.size(0) != L || !step_divides(a[4], B)) return not_plain();
  auto x = c10::make_intrusive<Extra>();
  dfa3d_problem &p = x->p;
  memset(&p, 0, sizeof p);
  if (!describe_dist(dist, B, dist.size(1), H, 0, 0, p)) return not_plain();
  p.B = (int32_t)B; p.N = (int32_t)dist.size(1); p.H = (int32_t)H; p.L = (int32_t)L; p.Q = (int32_t)Q; p.P = (int32_t)P;
  p.value_dtype = DFA3D_DTYPE_F32;
  Tensor r;
  {
    pybind11::gil_scoped_release nogil;
    r = wants_grad(dist, loc) ? DepthScoreFn::apply(dist, shapes, lsi, loc, x)
                              : depth_score_forward(p, dist, shapes, lsi, loc);
  }
  return THPVariable_Wrap(r);
}

PyObject *run_dist(PyObject *const *a, Py_ssize_t n) {
  // logits, shapes, lsi, num_pixels, activation code, storage code (DFA3D_DTYPE_*)
  if (n != 6 || !plain_mode()) return not_plain();
  Tensor logits, shapes, lsi;
  int64_t N, act, type;
  if (!float_tensor(a[0], logits, 4) || !long_tensor(a[1], shapes, 2) || !long_tensor(a[2], lsi, 1) || !integer(a[3], N) ||
      !integer(a[4], act) || !integer(a[5], type))
    return not_plain();
  if (!small(logits) || !one_device(logits, shapes, lsi) || (shapes.size(1) != 2 && shapes.size(1) != 3) ||
      lsi.size(0) != shapes.size(0) || N < 0 || N >= (int64_t(1) << 31))
    return not_plain();
  auto x = c10::make_intrusive<DistArgs>();
  x->N = (int32_t)N; x->act = (int32_t)act; x->dtype = (int32_t)type;
  const at::ScalarType st = type == DFA3D_DTYPE_F16 ? at::kHalf : type == DFA3D_DTYPE_BF16 ? at::kBFloat16 : at::kFloat;
  Tensor r;
  {
    pybind11::gil_scoped_release nogil;
    r = wants_grad(logits) ? DistFn::apply(logits, shapes, lsi, x, (int64_t)st)
                           : dist_forward(*x, logits, shapes, lsi, st);
  }
  return THPVariable_Wrap(r);
}

// bind({name: address}): the entry points of the loaded library
PyObject *py_bind(PyObject *, PyObject *table) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(PyDict_Check(table), "bind() takes a dict of addresses");
  auto get = [&](const char *name) {
    PyObject *o = PyDict_GetItemString(table, name);
    TORCH_CHECK(o != nullptr, "bind(): no address of ", name);
    return PyLong_AsVoidPtr(o);
  };
#define X(name) lib.name = reinterpret_cast<decltype(lib.name)>(get(#name));
  DFA3D_ENTRIES(X)
#undef X
  bound = true;
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

PyObject *py_entries(PyObject *, PyObject *) {
  static const char *names[] = {
#define X(name) #name,
      DFA3D_ENTRIES(X)
#undef X
  };
  PyObject *t = PyTuple_New(sizeof names / sizeof *names);
  for (size_t i = 0; i < sizeof names / sizeof *names; ++i) PyTuple_SET_ITEM(t, i, PyUnicode_FromString(names[i]));
  return t;
}

PyObject *py_calls(PyObject *, PyObject *) { return PyLong_FromLongLong(calls.load()); }

#define FAST(name, expr)                                                             \
  PyObject *py_##name(PyObject *, PyObject *const *a, Py_ssize_t n) {                 \
    HANDLE_TH_ERRORS                                                                  \
    return expr;                                                                      \
    END_HANDLE_TH_ERRORS                                                              \
  }
FAST(fused, run_fused(a, n, false, false))
FAST(fused_fp16, run_fused(a, n, false, true))
FAST(fused_ragged, run_fused(a, n, true, false))
FAST(attn3d, run_attn3d(a, n, false))
FAST(attn3d_ragged, run_attn3d(a, n, true))
FAST(attn3d_joint, run_attn3d_joint(a, n))
FAST(wms, run_attn2d(a, n, true, false))
FAST(wms_fp16, run_attn2d(a, n, true, true))
FAST(msda, run_attn2d(a, n, false, false))
FAST(msda_fp16, run_attn2d(a, n, false, true))
FAST(depth_score, run_depth_score(a, n))
FAST(dist_from_logits, run_dist(a, n))
#undef FAST

#define FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_##name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    {"bind", py_bind, METH_O, nullptr},
    {"entries", py_entries, METH_NOARGS, nullptr},
    {"calls", py_calls, METH_NOARGS, nullptr},
    FAST(fused), FAST(fused_fp16), FAST(fused_ragged), FAST(attn3d), FAST(attn3d_ragged), FAST(attn3d_joint),
    FAST(wms), FAST(wms_fp16),
    FAST(msda), FAST(msda_fp16), FAST(depth_score), FAST(dist_from_logits),
    {nullptr, nullptr, 0, nullptr},
};
#undef FAST

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) {
  PyObject *m = PyModule_Create(&module);
  // the headers this was compiled against: another torch may lay its classes out differently
  if (m && (PyModule_AddFunctions(m, dfa3d_torch::layer_methods) != 0 ||
            PyModule_AddStringConstant(m, "built_for", DFA3D_BUILT_FOR) != 0 ||
            PyModule_AddIntConstant(m, "split_rows", kSplitRows) != 0 || PyModule_AddIntConstant(m, "splits", kSplits) != 0)) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
