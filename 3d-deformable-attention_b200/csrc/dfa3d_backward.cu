// DFA3D backward kernels (sm_100a).
//
// Same decomposition as the forward: one warp per (camera, query, head) item, lane j owns sampling
// point j of a 32-point chunk.  Per chunk:
//   prologue -- the lane recomputes its point's geometry and per-corner depth scores from `dist`
//               (fused mode; the (B,Q,H,L,P,4) depth_score tensor is never read back) and publishes
//               {row offset, a * bilinear * depth score} per corner in shared memory;
//   rows     -- a group of G lanes reads one value row (4 channels per lane), takes its dot product with
//               the item's grad_out row (xor-shuffles inside the group) and adds
//               weight * grad_out to grad_value with one 16-byte vector reduction per lane
//               (red.global.add.v4.f32) instead of one scalar atomic per channel;
//   epilogue -- the four dot products t_k of a point return to its owner lane through shared
//               memory; grad_attn, grad_loc (x, y and, fused, z), grad_depth_score and the grad_dist
//               atomics all follow from t_k and the quantities the lane already holds.
// No block-wide barrier and no serial thread-0 reduction remain
// (cf. wms_deform_attn_cuda_kernel.cuh:378-407, ms_depth_score_sample_cuda_kernel.cuh:301-319).
#include "dfa3d_backward_point.cuh"
#include "dfa3d_launch.h"

namespace dfa3d {

// Softmax backward of the item's logits: grad_logit_j = a_j * (g_j - sum_k a_k g_k).  `partial` is the
// lane's share of the sum; the g_j were parked in grad_attn by the epilogue (each lane re-reads only
// what it wrote itself).
__device__ __forceinline__ void finish_logit_grads(const KArgs &a, const ItemCtx &c, int lane,
                                                   const SoftmaxStats &sm, float partial) {
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) partial += __shfl_xor_sync(0xffffffffu, partial, s);
  for (int j = lane; j < a.LP; j += 32) {
    float *g = a.grad_attn + (c.attn - a.attn) + j;
    const float aw = __fdiv_rn(expf(__ldg(c.attn + j) - sm.mx), sm.sum);
    *g = aw * (*g - partial);
  }
}

// One item of the backward: `table` / `dot_slots` are the warp's slices of shared memory.
template <typename VT, typename DT, int C, int MODE, bool FULL>
__device__ __forceinline__ void backward_item(const KArgs &a, const LevelTable &lv, const ItemCtx &c,
                                              RowEntry *table, float *dot_slots, int lane) {
  constexpr int V = RowVec4<VT>::kElems;
  constexpr int G = C / V;
  constexpr int R = 32 / G;
  constexpr int U = 4;
  // The table's slots past the last point hold no rows, and the dots of those are read by no one: a step may run over the
  // last point.  Conditions stand where the kernel comes out faster with them (20 points, 6 x 6000 queries x 8 heads, us
  // without / with): on the dots (from offsets, bf16 dist 906 / 892; two-stage of 16 channels 194 / 187) unless 16-bit rows
  // come with locations (648 / 666), on the rows for 16-bit rows with fp32 dist from offsets (831 / 806, 64 channels
  // 1236 / 1194; other types lose up to 5 %).
  constexpr bool kGuardDots = !FULL && !(MODE == kFused && sizeof(VT) == 2);
  constexpr bool kGuardRows = !FULL && MODE == kCallerFused && sizeof(VT) == 2 && sizeof(DT) == 4;
  const int sub = lane % G, grp = lane / G;
  const long long slice = ((long long)c.b * a.N * a.H + c.h) * C + sub * V;
  const VT *vbase = reinterpret_cast<const VT *>(a.value) + slice;
  float *gvbase = a.grad_value + slice;
  const RowEntry *my = table + grp;
  float *myd = dot_slots + grp;

  float go[V];
  {
    const float *gp = a.grad_out + (c.item * C + sub * V);
#pragma unroll
    for (int i = 0; i < V; i += 4) {
      const float4 t = __ldg(reinterpret_cast<const float4 *>(gp + i));
      go[i] = t.x; go[i + 1] = t.y; go[i + 2] = t.z; go[i + 3] = t.w;
    }
  }

  SoftmaxStats sm{0.f, 1.f};
  if (MODE == kCallerFused) sm = item_softmax_stats(a, c, lane);
  float dot = 0.f;

  for (int chunk = 0; chunk < a.LP; chunk += 32) {
    PointState st;
    float wgt[4];
    int off[4];
    bwd_point<DT, MODE>(a, lv, c, chunk + lane, sm, st, wgt, off);
    store_rows(table, lane, off, wgt);
    __syncwarp();
    const int nrows = FULL ? 128 : min(32, a.LP - chunk) * 4;
    auto step = [&](int r0) {
      RowEntry e[U];
      float v[U][V];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int r = r0 + u * R;
        e[u] = !kGuardRows || r + grp < nrows ? my[r] : RowEntry{-1, 0.f};
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (e[u].off >= 0) {
          RowVec4<VT>::load(vbase + e[u].off, v[u]);
        } else {
#pragma unroll
          for (int i = 0; i < V; ++i) v[u][i] = 0.f;
        }
      }
      float d[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        d[u] = 0.f;
#pragma unroll
        for (int i = 0; i < V; ++i) d[u] = fmaf(v[u][i], go[i], d[u]);
      }
      if (G >= 4) {
        int u_mine;
        const float f = fold_four_dots<G>(d, sub, u_mine);
        const int r = r0 + u_mine * R;
        if (u_mine >= 0 && (!kGuardDots || r + grp < nrows)) myd[r] = f;
      } else {
        // groups of 2 lanes (8 channels): a group's first lane stores its four totals one by one
#pragma unroll
        for (int u = 0; u < U; ++u) {
          float t = d[u];
#pragma unroll
          for (int s = 1; s < G; s <<= 1) t += __shfl_xor_sync(0xffffffffu, t, s);
          const int r = r0 + u * R;
          if (sub == 0 && (!kGuardDots || r + grp < nrows)) myd[r] = t;
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (e[u].off >= 0 && e[u].wgt != 0.f) {
          float *gp = gvbase + e[u].off;
#pragma unroll
          for (int i = 0; i < V; i += 4)
            red_add_v4(gp + i, e[u].wgt * go[i], e[u].wgt * go[i + 1], e[u].wgt * go[i + 2],
                       e[u].wgt * go[i + 3]);
        }
      }
    };
#pragma unroll 1
    for (int r0 = 0; r0 < nrows; r0 += R * U) step(r0);
    __syncwarp();
    const float4 tq = reinterpret_cast<const float4 *>(dot_slots)[lane];
    const float t[4] = {tq.x, tq.y, tq.z, tq.w};
    dot += bwd_point_epilogue<DT, MODE>(a, c, chunk + lane, st, t);
    __syncwarp();
  }
  if (MODE == kCallerFused) finish_logit_grads(a, c, lane, sm, dot);
}

// ------------------------------------------------------------------------------------------------
// fused / given-depth-score backward, C/4 a power of two
// ------------------------------------------------------------------------------------------------
// 4 CTAs (32 warps) per SM is the measured optimum (64 registers, a few bytes of spill); a CTA walks
// up to DFA3D_BWD_ITEMS_PER_WARP consecutive groups of 8 items before it retires.  WALK: that number; 0: a.rounds
// (dfa3d_walk.h), which costs registers that the kernel does not have (from offsets with bf16 dist 1202 us, 1194 as a constant).
template <typename VT, typename DT, int C, int MODE, bool FULL, int WALK>
__global__ void __launch_bounds__(kThreads, DFA3D_BWD_MIN_CTAS)
dfa3d_backward_kernel(const KArgs a) {
  __shared__ LevelTable lv;
  __shared__ __align__(16) RowEntry rows[kWarpsPerCta][128];
  __shared__ __align__(16) float dots[kWarpsPerCta][128];
  stage_levels(lv, a);
  const int rounds = WALK ? WALK : a.rounds, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll 1
  for (int it = 0; it < rounds; ++it) {
    ItemCtx c;
    if (!item_context<MODE, DFA3D_BWD_HEAD_MAJOR != 0>(a, warp, blockIdx.x * rounds + it, c)) return;
    backward_item<VT, DT, C, MODE, FULL>(a, lv, c, rows[warp], dots[warp], lane);
  }
}

// ------------------------------------------------------------------------------------------------
// any C: lanes stride over channels (correctness path for unusual widths)
// ------------------------------------------------------------------------------------------------
template <typename VT, typename DT, int MODE>
__global__ void __launch_bounds__(kThreads)
dfa3d_backward_generic_kernel(const KArgs a) {
  __shared__ LevelTable lv;
  __shared__ __align__(16) RowEntry rows[kWarpsPerCta][128];
  __shared__ __align__(16) float dots[kWarpsPerCta][128];
  stage_levels(lv, a);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  ItemCtx c;
  if (!item_context<MODE>(a, warp, blockIdx.x, c)) return;
  const int C = a.C;
  const long long slice = ((long long)c.b * a.N * a.H + c.h) * C;
  const VT *vbase = reinterpret_cast<const VT *>(a.value) + slice;
  float *gvbase = a.grad_value + slice;
  const float *gop = a.grad_out + c.item * C;
  RowEntry *my = rows[warp];
  float *myd = dots[warp];
  SoftmaxStats sm{0.f, 1.f};
  if (MODE == kCallerFused) sm = item_softmax_stats(a, c, lane);
  float dot = 0.f;
  for (int chunk = 0; chunk < a.LP; chunk += 32) {
    PointState st;
    float wgt[4];
    int off[4];
    bwd_point<DT, MODE>(a, lv, c, chunk + lane, sm, st, wgt, off);
    store_rows(my, lane, off, wgt);
    __syncwarp();
    const int nrows = min(32, a.LP - chunk) * 4;
    for (int r = 0; r < nrows; ++r) {
      const RowEntry e = my[r];
      float d = 0.f;
      if (e.off >= 0) {
        for (int ch = lane; ch < C; ch += 32) {
          const float g = __ldg(gop + ch);
          d = fmaf(load_scalar(vbase + e.off + ch), g, d);
          if (e.wgt != 0.f) red_add(gvbase + e.off + ch, e.wgt * g);
        }
      }
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) d += __shfl_xor_sync(0xffffffffu, d, s);
      if (lane == 0) myd[r] = d;
    }
    __syncwarp();
    const float4 tq = reinterpret_cast<const float4 *>(myd)[lane];
    const float t[4] = {tq.x, tq.y, tq.z, tq.w};
    dot += bwd_point_epilogue<DT, MODE>(a, c, chunk + lane, st, t);
    __syncwarp();
  }
  if (MODE == kCallerFused) finish_logit_grads(a, c, lane, sm, dot);
}

// ------------------------------------------------------------------------------------------------
// depth-score backward alone (two-stage API): one thread per sampling point
// ------------------------------------------------------------------------------------------------
template <typename DT>
__global__ void __launch_bounds__(kThreads)
dfa3d_depth_score_backward_kernel(const KArgs a) {
  __shared__ LevelTable lv;
  stage_levels(lv, a);
  const long long npts = a.items * a.LP;
  for (long long pt = (long long)blockIdx.x * blockDim.x + threadIdx.x; pt < npts;
       pt += (long long)gridDim.x * blockDim.x) {
    const long long item = pt / a.LP;
    const int j = (int)(pt - item * a.LP);
    const int l = j / a.P;
    const int h = (int)(item % a.H);
    const int b = (int)(item / a.items_per_cam);
    const float *lp = a.loc + pt * 3;
    const PointGeo g = point_geometry(__ldg(lp), __ldg(lp + 1), __ldg(lp + 2), true, lv.h[l], lv.w[l],
                                      lv.d[l], lv.start[l], a.N, dist_map_of(a, lv, l));
    float g_z = 0.f;
    if (g.ok3) {
      const long long bh = (long long)b * a.Nd * a.dist_pix_stride + h * a.dist_head_stride;
      const DT *dist_bh = reinterpret_cast<const DT *>(a.dist) + bh;
      float *gd_bh = a.grad_dist + bh;
      const float4 gq = __ldg(reinterpret_cast<const float4 *>(a.grad_ds_in) + pt);
      const float gds[4] = {gq.x, gq.y, gq.z, gq.w};
      const float hd = 1.f - g.ld;
      const int Dlim = min(g.Dd, a.D);
      float acc = 0.f;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (g.pix[k] >= 0) {
          float lo, hi;
          load_depth_pair(dist_bh, a.dist_pix_stride, g.dpix[k], g.z0, Dlim, true, lo, hi);
          red_depth_pair(gd_bh, a.dist_pix_stride, g.dpix[k], g.z0, Dlim, a.D, hd * gds[k], g.ld * gds[k]);
          acc = fmaf(gds[k], hi - lo, acc);
        }
      }
      g_z = (float)g.Dd * acc;
    }
    float *gl = a.grad_loc + pt * 3;
    gl[0] = 0.f; gl[1] = 0.f; gl[2] = g_z;
  }
}

// ------------------------------------------------------------------------------------------------
// host-side dispatch
// ------------------------------------------------------------------------------------------------
template <typename VT, typename DT, int C, int MODE, bool FULL>
static void launch_backward_c(KArgs &a, int cams, cudaStream_t s) {
  constexpr int kMost = DFA3D_BWD_ITEMS_PER_WARP;
  constexpr auto kLong = dfa3d_backward_kernel<VT, DT, C, MODE, FULL, kMost>;
  constexpr auto kShort = dfa3d_backward_kernel<VT, DT, C, MODE, FULL, 0>;
  a.rounds = walk_backward((a.items_per_cam + kWarpsPerCta - 1) / kWarpsPerCta, cams, kMost, resident_ctas<kLong>(), sm_count());
  const int per_cta = kWarpsPerCta * a.rounds;
  const dim3 grid((unsigned)((a.items_per_cam + per_cta - 1) / per_cta), (unsigned)cams, 1);
  if (a.rounds == kMost) kLong<<<grid, kThreads, 0, s>>>(a);
  else kShort<<<grid, kThreads, 0, s>>>(a);
}

template <typename VT, typename DT, int MODE, bool FULL>
static void launch_backward_g(KArgs &a, int cams, cudaStream_t s) {
  constexpr int V = RowVec4<VT>::kElems;
  switch ((a.C % V == 0) ? a.C / V : 0) {
    case 2:  launch_backward_c<VT, DT, 2 * V, MODE, FULL>(a, cams, s); break;
    case 4:  launch_backward_c<VT, DT, 4 * V, MODE, FULL>(a, cams, s); break;
    case 8:  launch_backward_c<VT, DT, 8 * V, MODE, FULL>(a, cams, s); break;
    case 16: launch_backward_c<VT, DT, 16 * V, MODE, FULL>(a, cams, s); break;
    case 32: launch_backward_c<VT, DT, 32 * V, MODE, FULL>(a, cams, s); break;
    default: {
      const dim3 g1((unsigned)((a.items_per_cam + kWarpsPerCta - 1) / kWarpsPerCta), (unsigned)cams, 1);
      dfa3d_backward_generic_kernel<VT, DT, MODE><<<g1, kThreads, 0, s>>>(a);
      break;
    }
  }
}

template <typename VT, typename DT, int MODE>
static cudaError_t launch_backward_vd(const KArgs &a0, cudaStream_t s) {
  for (int b0 = 0; b0 < a0.B; b0 += 65535) {      // grid.y limit
    KArgs a = a0;
    a.b0 = b0;
    const int cams = min(65535, a0.B - b0);
    if (a.LP % 32 == 0) launch_backward_g<VT, DT, MODE, true>(a, cams, s);
    else launch_backward_g<VT, DT, MODE, false>(a, cams, s);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// Storage types are the DFA3D_DTYPE_* codes of the C header.  fp32 and bf16 combine freely; fp16 value
// goes with fp16 dist (what a half-precision caller passes) -- the C entry points reject the rest.
template <int MODE>
static cudaError_t launch_backward_m(const KArgs &a, int value_dtype, int dist_dtype, cudaStream_t s) {
  if (value_dtype == kDtypeF16) return launch_backward_vd<__half, __half, MODE>(a, s);
  if (value_dtype == kDtypeBF16)
    return dist_dtype == kDtypeBF16 ? launch_backward_vd<__nv_bfloat16, __nv_bfloat16, MODE>(a, s)
                                    : launch_backward_vd<__nv_bfloat16, float, MODE>(a, s);
  return dist_dtype == kDtypeBF16 ? launch_backward_vd<float, __nv_bfloat16, MODE>(a, s)
                                  : launch_backward_vd<float, float, MODE>(a, s);
}

cudaError_t launch_backward(const KArgs &a, int value_dtype, int dist_dtype, int mode, cudaStream_t s) {
  if (a.items == 0) return cudaSuccess;
  if (packed_covers(a.LP, a.C)) return launch_backward_packed(a, value_dtype, dist_dtype, mode, s);
  if (mode == kCallerFused2D) return cudaErrorNotSupported;       // see attn2d_supported
  if (mode == kGivenDepthScore) {
    if (value_dtype == kDtypeF16) return launch_backward_vd<__half, float, kGivenDepthScore>(a, s);
    return value_dtype == kDtypeBF16 ? launch_backward_vd<__nv_bfloat16, float, kGivenDepthScore>(a, s)
                                     : launch_backward_vd<float, float, kGivenDepthScore>(a, s);
  }
  if (mode == kCallerFused) return launch_backward_m<kCallerFused>(a, value_dtype, dist_dtype, s);
  return launch_backward_m<kFused>(a, value_dtype, dist_dtype, s);
}

cudaError_t launch_depth_score_backward(const KArgs &a, int dist_dtype, cudaStream_t s) {
  const long long npts = a.items * a.LP;
  if (npts == 0) return cudaSuccess;
  const unsigned grid = (unsigned)min((npts + kThreads - 1) / kThreads, (long long)148 * 64);
  if (dist_dtype == kDtypeF16) dfa3d_depth_score_backward_kernel<__half><<<grid, kThreads, 0, s>>>(a);
  else if (dist_dtype == kDtypeBF16) dfa3d_depth_score_backward_kernel<__nv_bfloat16><<<grid, kThreads, 0, s>>>(a);
  else dfa3d_depth_score_backward_kernel<float><<<grid, kThreads, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace dfa3d
