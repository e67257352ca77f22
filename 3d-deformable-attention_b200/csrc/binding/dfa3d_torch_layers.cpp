// Native host path of the layer around the operator: Linear (with or without a ReLU, and three of one input), residual
// add + LayerNorm, the re-batching of queries, and 2-D attention from offsets and logits.  Same contract as
// dfa3d_torch.cpp: NotImplemented means that the Python code has to take the call.
#include "dfa3d_torch.h"

using namespace dfa3d_torch;

namespace {

// ------------------------------------------------------------------------------------------------
// Linear
// ------------------------------------------------------------------------------------------------
Tensor rows_of(const Tensor &t) { return t.view({-1, t.size(-1)}); }

// Weight gradient g^T x of g (rows, out) and x (rows, in), and bias gradient: the column sums of g.  Many rows into a small
// product is one long reduction that cuBLAS gives to few CTAs; as a batch of 16 row slices, summed by a kernel of our own
// that also takes the rows left over and zeroes the bias gradient, it takes a third of the time.
void parameter_gradients(const Tensor &g, const Tensor &x, bool weight, bool bias, Tensor &gw, Tensor &gb) {
  const int64_t rows = g.size(0), out = g.size(1), in = x.size(1);
  void *s = stream_of(g);
  if (bias) gb = empty_f32({out}, g);
  bool zeroed = false;
  if (weight && (rows < kSplitRows || in % 4 != 0)) {
    gw = at::mm(g.t(), x);
  } else if (weight) {
    const int64_t k = rows / kSplits, head = k * kSplits;
    const Tensor part = at::bmm(g.as_strided({kSplits, out, k}, {k * out, 1, out}), x.as_strided({kSplits, k, in}, {k * in, in, 1}));
    gw = empty_f32({out, in}, g);
    const bool own_tail = aligned(x, 16);             // the kernel reads x's last rows in 16-byte words
    check(lib.dfa3d_slice_sum(fp(part), (int32_t)kSplits, (int32_t)out, (int32_t)in, fp(g) + head * out, fp(x) + head * in,
                              own_tail ? (int32_t)(rows - head) : 0, fpm(gw), bias ? fpm(gb) : nullptr, s),
          "dfa3d_slice_sum");
    if (!own_tail && head < rows) gw.addmm_(g.narrow(0, head, rows - head).t(), x.narrow(0, head, rows - head));
    zeroed = true;
  }
  if (!bias) return;
  if (!zeroed) zero_two(gb, Tensor(), s);
  check(lib.dfa3d_column_sum(fp(g), rows, (int32_t)out, fpm(gb), s), "dfa3d_column_sum");
}

Tensor linear_forward(const Tensor &x, const Tensor &w, const Tensor &b, bool relu) {
  std::vector<int64_t> sz(x.sizes().begin(), x.sizes().end());
  sz.back() = w.size(0);
  Tensor y = at::empty(sz, x.options());
  Tensor y2 = rows_of(y);
  if (relu) at::_addmm_activation_out(y2, b, rows_of(x), w.t(), 1, 1, false);
  else at::addmm_out(y2, b, rows_of(x), w.t());
  return y;
}

// The products of a backward are of the forward's kind, float32, wherever backward() is called: autograd carries the caller's
// autocast state into the node, where a product in 16 bits would be taken for a float32 one.
using NoAutocast = c10::impl::ExcludeDispatchKeyGuard;

struct LinearFn : torch::autograd::Function<LinearFn> {
  static Tensor forward(AutogradContext *ctx, const Tensor &x, const Tensor &w, const Tensor &b, bool relu) {
    c10::cuda::CUDAGuard guard(x.device());
    Tensor y = linear_forward(x, w, b, relu);
    keep(ctx, c10::make_intrusive<Kept>(), {x, w, relu ? y : Tensor()});
    return y;
  }
  static variable_list backward(AutogradContext *ctx, variable_list grads) {
    const NoAutocast no_autocast(c10::autocast_dispatch_keyset);
    variable_list v;
    kept<Kept>(ctx, v);
    const Tensor &x = v[0], &w = v[1];
    c10::cuda::CUDAGuard guard(x.device());
    Tensor g = rows_of(f32(grads[0])), gx, gw, gb;
    const bool relu = v[2].defined();
    if (relu) {
      void *s = stream_of(g);
      if (!aligned(g, 16)) g = g.clone();
      Tensor masked = at::empty_like(g);
      gb = empty_f32({g.size(1)}, g);
      zero_two(gb, Tensor(), s);
      check(lib.dfa3d_relu_backward_column_sum(fp(g), fp(v[2]), g.size(0), (int32_t)g.size(1), fpm(masked), fpm(gb), s),
            "dfa3d_relu_backward_column_sum");
      g = masked;
    }
    if (ctx->needs_input_grad(0)) gx = at::mm(g, w).view(x.sizes());
    Tensor none;
    parameter_gradients(g, rows_of(x), ctx->needs_input_grad(1), !relu && ctx->needs_input_grad(2), gw, relu ? none : gb);
    return once({gx, gw, gb, Tensor()}, grads);
  }
};

// Two or three Linear layers of one input, run as one with their weights one below the other: y = [y0 | y1 | y2].  One
// product instead of three each way, one pass over y's gradient for the bias, and the input's gradient is not summed up
// from parts.
struct JointLinearFn : torch::autograd::Function<JointLinearFn> {
  static Tensor forward(AutogradContext *ctx, const Tensor &x, const Tensor &w0, const Tensor &b0, const Tensor &w1,
                        const Tensor &b1, const std::optional<Tensor> &w2, const std::optional<Tensor> &b2) {
    c10::cuda::CUDAGuard guard(x.device());
    const Tensor *w[3] = {&w0, &w1, w2 ? &*w2 : nullptr}, *b[3] = {&b0, &b1, b2 ? &*b2 : nullptr};
    const int n = w2 ? 3 : 2;
    int64_t out = 0, counts[6];
    std::vector<int64_t> split;
    for (int i = 0; i < n; ++i) {
      split.push_back(w[i]->size(0));
      out += w[i]->size(0);
    }
    Tensor W = at::empty({out, x.size(-1)}, x.options()), B = at::empty({out}, x.options());
    const float *src[6];
    float *dst[6], *wd = fpm(W), *bd = fpm(B);
    for (int i = 0; i < n; ++i) {
      src[i] = fp(*w[i]); dst[i] = wd; counts[i] = w[i]->numel();
      src[n + i] = fp(*b[i]); dst[n + i] = bd; counts[n + i] = b[i]->numel();
      wd += counts[i]; bd += counts[n + i];
    }
    check(lib.dfa3d_copy_segments(src, dst, counts, 2 * n, stream_of(x)), "dfa3d_copy_segments");
    keep(ctx, c10::make_intrusive<Kept>(), {x, W});
    ctx->saved_data["split"] = split;
    return linear_forward(x, W, B, false);
  }
  static variable_list backward(AutogradContext *ctx, variable_list grads) {
    const NoAutocast no_autocast(c10::autocast_dispatch_keyset);
    variable_list v;
    kept<Kept>(ctx, v);
    const Tensor &x = v[0], &W = v[1];
    c10::cuda::CUDAGuard guard(x.device());
    const Tensor g = rows_of(f32(grads[0]));
    const auto split = ctx->saved_data["split"].toIntVector();
    variable_list out(7);
    bool weight = false, bias = false;
    for (size_t i = 0; i < split.size(); ++i) {
      weight |= ctx->needs_input_grad(1 + 2 * i);
      bias |= ctx->needs_input_grad(2 + 2 * i);
    }
    if (ctx->needs_input_grad(0)) out[0] = at::mm(g, W).view(x.sizes());
    Tensor gw, gb;
    parameter_gradients(g, rows_of(x), weight, bias, gw, gb);
    int64_t at = 0;
    for (size_t i = 0; i < split.size(); ++i) {
      if (ctx->needs_input_grad(1 + 2 * i)) out[1 + 2 * i] = gw.narrow(0, at, split[i]);
      if (ctx->needs_input_grad(2 + 2 * i)) out[2 + 2 * i] = gb.narrow(0, at, split[i]);
      at += split[i];
    }
    return once(std::move(out), grads);
  }
};

bool linear_arguments(PyObject *const *a, const Tensor &x, Tensor &w, Tensor &b) {
  return float_tensor(a[0], w, 2) && float_tensor(a[1], b, 1) && one_device(x, w, b) && w.size(1) == x.size(-1) &&
         b.size(0) == w.size(0) && w.size(0) % 4 == 0 && w.size(0) > 0;
}

PyObject *run_linear(PyObject *const *a, Py_ssize_t n, bool relu) {
  if (n != 3 || !plain_mode()) return not_plain();
  Tensor x, w, b;
  if (!float_tensor(a[0], x, -1) || x.dim() < 1 || x.numel() == 0 || !linear_arguments(a + 1, x, w, b)) return not_plain();
  Tensor y;
  {
    pybind11::gil_scoped_release nogil;
    if (wants_grad(x, w, b)) {
      y = LinearFn::apply(x, w, b, relu);
    } else {
      c10::cuda::CUDAGuard guard(x.device());
      y = linear_forward(x, w, b, relu);
    }
  }
  return THPVariable_Wrap(y);
}

PyObject *run_joint_linear(PyObject *const *a, Py_ssize_t n) {
  // x, w0, b0, w1, b1 [, w2, b2]
  if ((n != 5 && n != 7) || !plain_mode()) return not_plain();
  Tensor x, w[3], b[3];
  if (!float_tensor(a[0], x, -1) || x.dim() < 1 || x.numel() == 0) return not_plain();
  for (int i = 0; i < (n - 1) / 2; ++i)
    if (!linear_arguments(a + 1 + 2 * i, x, w[i], b[i])) return not_plain();
  Tensor y;
  {
    pybind11::gil_scoped_release nogil;
    y = JointLinearFn::apply(x, w[0], b[0], w[1], b[1], given(w[2]), given(b[2]));
  }
  return THPVariable_Wrap(y);
}

// ------------------------------------------------------------------------------------------------
// residual add + LayerNorm
// ------------------------------------------------------------------------------------------------
struct AddLayerNormFn : torch::autograd::Function<AddLayerNormFn> {
  static Tensor forward(AutogradContext *ctx, const Tensor &x, const std::optional<Tensor> &res, const Tensor &w,
                        const Tensor &b, double eps) {
    c10::cuda::CUDAGuard guard(x.device());
    const int64_t E = x.size(-1), rows = x.numel() / E;
    Tensor y = at::empty_like(x), sum, stats = empty_f32({2, rows}, x);
    if (res) sum = at::empty_like(x);
    float *mean = fpm(stats), *rstd = mean + rows;
    check(lib.dfa3d_add_layer_norm_forward(fp(x), res ? fp(*res) : nullptr, fp(w), fp(b), rows, (int32_t)E, (float)eps,
                                           res ? fpm(sum) : nullptr, fpm(y), mean, rstd, stream_of(x)),
          "dfa3d_add_layer_norm_forward");
    keep(ctx, c10::make_intrusive<Kept>(), {res ? sum : x, w, stats});
    ctx->saved_data["res"] = res.has_value();
    return y;
  }
  static variable_list backward(AutogradContext *ctx, variable_list grads) {
    variable_list v;
    kept<Kept>(ctx, v);
    const Tensor &in = v[0], &w = v[1], &stats = v[2];
    c10::cuda::CUDAGuard guard(in.device());
    const int64_t E = in.size(-1), rows = in.numel() / E;
    const Tensor g = f32(grads[0]);
    void *s = stream_of(in);
    Tensor gin = at::empty_like(in), gw = empty_f32({E}, in), gb = empty_f32({E}, in);
    zero_two(gw, gb, s);
    check(lib.dfa3d_layer_norm_backward(fp(g), fp(in), fp(w), fp(stats), fp(stats) + rows, rows, (int32_t)E, fpm(gin), fpm(gw),
                                        fpm(gb), s),
          "dfa3d_layer_norm_backward");
    return once({gin, ctx->saved_data["res"].toBool() ? gin : Tensor(), gw, gb, Tensor()}, grads);
  }
};

PyObject *run_add_layer_norm(PyObject *const *a, Py_ssize_t n) {
  // x, residual or None, weight, bias, eps
  if (n != 5 || !plain_mode() || !PyFloat_CheckExact(a[4])) return not_plain();
  Tensor x, res, w, b;
  const bool with = a[1] != Py_None;
  if (!float_tensor(a[0], x, -1) || x.dim() < 1 || x.numel() == 0 || (with && !float_tensor(a[1], res, -1)) ||
      !float_tensor(a[2], w, 1) || !float_tensor(a[3], b, 1))
    return not_plain();
  const int64_t E = x.size(-1);
  if (w.numel() != E || b.numel() != E || E % 4 != 0 || E > 1024 || !one_device(x, w, b) ||
      (with && (res.sizes() != x.sizes() || !one_device(x, res))))
    return not_plain();
  const double eps = PyFloat_AS_DOUBLE(a[4]);
  Tensor y;
  {
    pybind11::gil_scoped_release nogil;
    if (wants_grad(x, w, b) || (with && wants_grad(res))) {
      y = AddLayerNormFn::apply(x, with ? std::optional<Tensor>(res) : std::nullopt, w, b, eps);
    } else {
      c10::cuda::CUDAGuard guard(x.device());
      y = at::empty_like(x);
      check(lib.dfa3d_add_layer_norm_infer(fp(x), with ? fp(res) : nullptr, fp(w), fp(b), x.numel() / E, (int32_t)E,
                                           (float)eps, fpm(y), stream_of(x)),
            "dfa3d_add_layer_norm_infer");
    }
  }
  return THPVariable_Wrap(y);
}

// ------------------------------------------------------------------------------------------------
// re-batching
// ------------------------------------------------------------------------------------------------
struct PlanRef : torch::CustomClassHolder {
  Tensor query, camera, offsets, row_of, inv_count;
  int64_t cams = 0, bs = 0, Q = 0, rows = 0;
};

// packed_query, packed_camera, offsets, row_of, inv_count, cams, bs, Q, rows
bool plan_arguments(PyObject *const *a, PlanRef &p) {
  auto ints = [](PyObject *o, Tensor &t) { return plain_tensor(o, t) && t.scalar_type() == at::kInt; };
  return ints(a[0], p.query) && ints(a[1], p.camera) && ints(a[2], p.offsets) && ints(a[3], p.row_of) &&
         float_tensor(a[4], p.inv_count, 2) && integer(a[5], p.cams) && integer(a[6], p.bs) && integer(a[7], p.Q) &&
         integer(a[8], p.rows);
}
constexpr int kPlanArguments = 9;

Tensor plan_gather(const PlanRef &p, const Tensor &src, int64_t width, int64_t cam_stride, int64_t batch_stride, bool scaled) {
  Tensor dst = empty_f32({p.bs * p.rows, width}, src);
  check(lib.dfa3d_rebatch_gather(fp(src), ip(p.query), ip(p.camera), ip(p.offsets), (int32_t)p.cams, (int32_t)p.bs,
                                 (int32_t)p.Q, (int32_t)width, cam_stride, batch_stride, scaled ? fp(p.inv_count) : nullptr,
                                 fpm(dst), p.bs * p.rows, stream_of(src)),
        "dfa3d_rebatch_gather");
  return dst;
}

Tensor plan_combine(const PlanRef &p, const Tensor &packed, int64_t width, bool scaled) {
  Tensor dst = empty_f32({p.bs, p.Q, width}, packed);
  check(lib.dfa3d_rebatch_combine(packed.numel() ? fp(packed) : fp(p.inv_count), ip(p.row_of), ip(p.offsets), (int32_t)p.cams,
                                  (int32_t)p.bs, (int32_t)p.Q, (int32_t)width, scaled ? fp(p.inv_count) : nullptr, fpm(dst),
                                  stream_of(packed)),
        "dfa3d_rebatch_combine");
  return dst;
}

struct GatherFn : torch::autograd::Function<GatherFn> {
  static Tensor forward(AutogradContext *ctx, const Tensor &src, c10::intrusive_ptr<PlanRef> p) {
    c10::cuda::CUDAGuard guard(src.device());
    ctx->saved_data["p"] = c10::IValue::make_capsule(p);
    return plan_gather(*p, src, src.size(2), 0, p->Q, false);
  }
  static variable_list backward(AutogradContext *ctx, variable_list grads) {
    const auto p = c10::static_intrusive_pointer_cast<PlanRef>(ctx->saved_data.at("p").toCapsule());
    c10::cuda::CUDAGuard guard(grads[0].device());
    const Tensor g = f32(grads[0]);
    return once({plan_combine(*p, g, g.size(1), false), Tensor()}, grads);
  }
};

struct CombineFn : torch::autograd::Function<CombineFn> {
  static Tensor forward(AutogradContext *ctx, const Tensor &packed, c10::intrusive_ptr<PlanRef> p) {
    c10::cuda::CUDAGuard guard(packed.device());
    ctx->saved_data["p"] = c10::IValue::make_capsule(p);
    return plan_combine(*p, packed, packed.size(1), true);
  }
  static variable_list backward(AutogradContext *ctx, variable_list grads) {
    const auto p = c10::static_intrusive_pointer_cast<PlanRef>(ctx->saved_data.at("p").toCapsule());
    c10::cuda::CUDAGuard guard(grads[0].device());
    const Tensor g = f32(grads[0]);
    return once({plan_gather(*p, g, g.size(2), 0, p->Q, true), Tensor()}, grads);
  }
};

PyObject *run_gather(PyObject *const *a, Py_ssize_t n) {
  // src (bs, Q, W), plan
  if (n != 1 + kPlanArguments || !plain_mode()) return not_plain();
  auto p = c10::make_intrusive<PlanRef>();
  Tensor src;
  if (!float_tensor(a[0], src, 3) || !plan_arguments(a + 1, *p) || src.size(0) != p->bs || src.size(1) != p->Q ||
      !one_device(src, p->query) || src.size(2) <= 0 || src.size(2) >= (1 << 24))
    return not_plain();
  Tensor r;
  {
    pybind11::gil_scoped_release nogil;
    if (wants_grad(src)) {
      r = GatherFn::apply(src, p);
    } else {
      c10::cuda::CUDAGuard guard(src.device());
      r = plan_gather(*p, src, src.size(2), 0, p->Q, false);
    }
  }
  return THPVariable_Wrap(r);
}

PyObject *run_combine(PyObject *const *a, Py_ssize_t n) {
  // packed (bs*rows, W), plan
  if (n != 1 + kPlanArguments || !plain_mode()) return not_plain();
  auto p = c10::make_intrusive<PlanRef>();
  Tensor packed;
  if (!float_tensor(a[0], packed, 2) || !plan_arguments(a + 1, *p) || packed.size(0) != p->bs * p->rows ||
      !one_device(packed, p->query) || packed.size(1) <= 0 || packed.size(1) >= (1 << 24))
    return not_plain();
  Tensor r;
  {
    pybind11::gil_scoped_release nogil;
    if (wants_grad(packed)) {
      r = CombineFn::apply(packed, p);
    } else {
      c10::cuda::CUDAGuard guard(packed.device());
      r = plan_combine(*p, packed, packed.size(1), true);
    }
  }
  return THPVariable_Wrap(r);
}

PyObject *run_gather_per_camera(PyObject *const *a, Py_ssize_t n) {
  // src (cams, bs, Q, ...) without gradient, plan
  if (n != 1 + kPlanArguments || !plain_mode()) return not_plain();
  PlanRef p;
  Tensor src;
  if (!float_tensor(a[0], src, -1) || src.dim() < 4 || !plan_arguments(a + 1, p) || src.size(0) != p.cams ||
      src.size(1) != p.bs || src.size(2) != p.Q || !one_device(src, p.query) || src.numel() == 0)
    return not_plain();
  Tensor r;
  {
    pybind11::gil_scoped_release nogil;
    at::NoGradGuard none;
    c10::cuda::CUDAGuard guard(src.device());
    std::vector<int64_t> sz{p.bs * p.rows};
    int64_t width = 1;
    for (int64_t i = 3; i < src.dim(); ++i) {
      sz.push_back(src.size(i));
      width *= src.size(i);
    }
    r = plan_gather(p, src, width, p.bs * p.Q, p.Q, false).view(sz);
  }
  return THPVariable_Wrap(r);
}

// ------------------------------------------------------------------------------------------------
// 2-D attention from offsets and logits side by side in one row per query
// ------------------------------------------------------------------------------------------------
struct Attn2dExtra : Kept {
  dfa3d_problem p;
  int32_t maps = 1;
};

// Rows of `joint`: offsets, then logits.
Tensor attn2d_forward(const Attn2dExtra &x, const Tensor &value, const Tensor &shapes, const Tensor &lsi, const Tensor &ref,
                      const Tensor &joint) {
  c10::cuda::CUDAGuard guard(value.device());
  const int64_t row = joint.size(-1);
  Tensor out = empty_f32({x.p.B, x.p.Q, (int64_t)x.p.H * x.p.C}, value);
  check(lib.dfa3d_attn2d_forward(&x.p, x.maps, row, row, value.const_data_ptr(), lp(shapes), lp(lsi), fp(ref), fp(joint),
                                 fp(joint) + row / 3 * 2, fpm(out), stream_of(value)),
        "dfa3d_attn2d_forward");
  return out;
}

struct Attn2dFn : torch::autograd::Function<Attn2dFn> {
  static Tensor forward(AutogradContext *ctx, const Tensor &value, const Tensor &shapes, const Tensor &lsi,
                        const Tensor &ref, const Tensor &joint, c10::intrusive_ptr<Attn2dExtra> x) {
    keep(ctx, x, {value, shapes, lsi, ref, joint});
    return attn2d_forward(*x, value, shapes, lsi, ref, joint);
  }
  static variable_list backward(AutogradContext *ctx, variable_list grads) {
    variable_list v;
    const auto x = kept<Attn2dExtra>(ctx, v);
    const Tensor &value = v[0], &joint = v[4];
    c10::cuda::CUDAGuard guard(value.device());
    const Tensor go = f32(grads[0]);
    Tensor gv = at::empty_like(value), gj = at::empty_like(joint);
    const int64_t row = joint.size(-1), logits = row / 3 * 2;
    void *s = stream_of(value);
    zero_two(gv, Tensor(), s);
    check(lib.dfa3d_attn2d_backward(&x->p, x->maps, row, row, value.const_data_ptr(), lp(v[1]), lp(v[2]), fp(v[3]), fp(joint),
                                    fp(joint) + logits, fp(go), fpm(gv), fpm(gj), fpm(gj) + logits, s),
          "dfa3d_attn2d_backward");
    return once({gv, Tensor(), Tensor(), Tensor(), gj, Tensor()}, grads);
  }
};

PyObject *run_attn2d(PyObject *const *a, Py_ssize_t n) {
  // value (bs*maps, N, H*C), shapes (L, 2), lsi (L), ref (bs*maps, Q, L, 2), joint (bs, Q, H*maps*L*P*3), maps, heads, points
  int64_t maps, H, P;
  if (n != 8 || !plain_mode() || !integer(a[5], maps) || !integer(a[6], H) || !integer(a[7], P)) return not_plain();
  Tensor value, shapes, lsi, ref, joint;
  if (!float_tensor(a[0], value, 3) || !long_tensor(a[1], shapes, 2) || !long_tensor(a[2], lsi, 1) ||
      !float_tensor(a[3], ref, 4) || !float_tensor(a[4], joint, 3))
    return not_plain();
  if (maps <= 0 || H <= 0 || P <= 0 || maps > 16 || value.size(2) % H != 0 || value.size(0) % maps != 0 || !small(value) ||
      !small(joint) || !one_device(value, shapes, lsi, ref, joint) || ref.requires_grad())
    return not_plain();
  if (!aligned(value, 16) || !aligned(ref, 8) || !aligned(joint, 8)) return not_plain();
  const int64_t bs = value.size(0) / maps, Q = joint.size(1), L = shapes.size(0), pts = H * maps * L * P;
  if (shapes.size(1) != 2 || lsi.size(0) != L || !sizes_are(ref, {bs * maps, Q, L, 2}) || !sizes_are(joint, {bs, Q, pts * 3}))
    return not_plain();
  auto x = c10::make_intrusive<Attn2dExtra>();
  dfa3d_problem &p = x->p;
  memset(&p, 0, sizeof p);
  p.B = (int32_t)bs; p.N = (int32_t)value.size(1); p.H = (int32_t)H; p.C = (int32_t)(value.size(2) / H);
  p.D = 1; p.L = (int32_t)L; p.Q = (int32_t)Q; p.P = (int32_t)P;
  p.value_dtype = p.dist_dtype = DFA3D_DTYPE_F32;
  x->maps = (int32_t)maps;
  if (!lib.dfa3d_attn2d_supported(&p, x->maps)) return not_plain();
  Tensor r;
  {
    pybind11::gil_scoped_release nogil;
    r = wants_grad(value, joint) ? Attn2dFn::apply(value, shapes, lsi, ref, joint, x)
                                 : attn2d_forward(*x, value, shapes, lsi, ref, joint);
  }
  return THPVariable_Wrap(r);
}

#define FAST(name, expr)                                                             \
  PyObject *py_##name(PyObject *, PyObject *const *a, Py_ssize_t n) {                 \
    HANDLE_TH_ERRORS                                                                  \
    return expr;                                                                      \
    END_HANDLE_TH_ERRORS                                                              \
  }
FAST(linear, run_linear(a, n, false))
FAST(linear_relu, run_linear(a, n, true))
FAST(joint_linear, run_joint_linear(a, n))
FAST(add_layer_norm, run_add_layer_norm(a, n))
FAST(gather_queries, run_gather(a, n))
FAST(combine_cameras, run_combine(a, n))
FAST(gather_per_camera, run_gather_per_camera(a, n))
FAST(attn2d, run_attn2d(a, n))
#undef FAST

}  // namespace

namespace dfa3d_torch {
#define FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_##name)), METH_FASTCALL, nullptr}
PyMethodDef layer_methods[] = {
    FAST(linear), FAST(linear_relu), FAST(joint_linear), FAST(add_layer_norm), FAST(gather_queries), FAST(combine_cameras),
    FAST(gather_per_camera), FAST(attn2d), {nullptr, nullptr, 0, nullptr},
};
#undef FAST
}  // namespace dfa3d_torch
