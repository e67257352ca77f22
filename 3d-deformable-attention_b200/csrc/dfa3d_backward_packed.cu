// DFA3D backward for items of few points (L*P <= 16): a warp takes several consecutive items at once (sm_100a).
//
// An item has LPP lanes -- 4, 8 or 16 (packed_lanes) -- and lane j of them owns its point j (full or nearly
// full, coalesced prologue and epilogue); a group of G lanes walks the rows of one item -- or a share of them when the warp
// holds fewer items than groups -- with that item's grad_out fragment.  Same row phase as the one-item kernels otherwise,
// and the same bound: the row reductions, in L2 and on the way to it.
#include "dfa3d_backward_point.cuh"
#include "dfa3d_launch.h"

namespace dfa3d {
namespace {

// The row loop is not unrolled: its ends vary, and unrolled it spilled (1 level x 8 points, 6 x 6000 queries: 310 us
// unrolled, 291 like this; head-major order, 3 or 5 CTAs per SM and reductions before the dot products: within 2 %).
template <typename VT, typename DT, int C, int MODE, int LPP>
__global__ void __launch_bounds__(kThreads, DFA3D_BWD_MIN_CTAS)
dfa3d_backward_packed_kernel(const KArgs a) {
  constexpr int V = RowVec4<VT>::kElems;
  constexpr int G = C / V;
  constexpr int R = 32 / G;
  constexpr int K = 32 / LPP;
  constexpr int GPI = R > K ? R / K : 1;
  constexpr int IPG = K > R ? K / R : 1;
  constexpr int U = 4;
  constexpr int kSlots = LPP * 4;              // row slots of one item
  static_assert(G >= 4 && 32 % LPP == 0 && 32 % G == 0 && kSlots % (GPI * U) == 0, "unsupported packing");
  __shared__ LevelTable lv;
  __shared__ __align__(16) RowEntry rows[kWarpsPerCta][128];
  __shared__ __align__(16) float dots[kWarpsPerCta][128];
  stage_levels(lv, a);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane % G, grp = lane / G;
  const int b = (int)blockIdx.y + a.b0;
  const long long cam = (long long)b * a.N * a.H * C + sub * V;
  const VT *vbase = reinterpret_cast<const VT *>(a.value) + cam;
  float *gvbase = a.grad_value + cam;
  RowEntry *table = rows[warp];
  float *dot_slots = dots[warp];
  // the camera's queries: rows [q0, q0 + nq) of the per-query tensors
  const long long q0 = a.q_off ? (long long)__ldg(a.q_off + b) : (long long)b * a.Q;
  const unsigned nitems = (unsigned)(a.q_off ? __ldg(a.q_off + b + 1) - (int)q0 : a.Q) * (unsigned)a.H;
  const int nrows = a.LP * 4;
#pragma unroll 1
  for (int it = 0; it < a.rounds; ++it) {
    const unsigned first = ((blockIdx.x * a.rounds + it) * kWarpsPerCta + warp) * K;
    if (first >= nitems) return;
    const unsigned idx = first + lane / LPP;
    const bool live = idx < nitems && lane % LPP < a.LP;
    ItemCtx c;
    c.b = b;
    {
      const unsigned q = idx / (unsigned)a.H;
      c.h = (int)(idx - q * (unsigned)a.H);
      c.bq = q0 + q;
    }
    c.item = q0 * a.H + idx;
    item_inputs<MODE>(a, c);
    const int j = live ? lane % LPP : a.LP;      // a.LP: no such point, the lane stays idle
    SoftmaxStats sm{0.f, 1.f};
    // lanes of a softmax: the item's, in 2-D those of one map
    const int lanes = MODE == kCallerFused2D ? LPP / a.maps : LPP;
    if (mode_from_offsets(MODE)) sm = lanes_softmax_stats(live ? __ldg(c.attn + j) : 0.f, live, lanes);
    PointState st;
    {
      float wgt[4];
      int off[4];
      bwd_point<DT, MODE>(a, lv, c, j, sm, st, wgt, off);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (off[k] >= 0) off[k] += c.h * C;
      store_rows(table, lane, off, wgt);
    }
    __syncwarp();
#pragma unroll
    for (int t = 0; t < IPG; ++t) {
      const int i = grp / GPI + t * (R / GPI);
      const unsigned item_i = first + i;
      const int base = i * kSlots + (grp % GPI) * U;
      float go[V];
      if (item_i < nitems) {
        const float *gp = a.grad_out + ((q0 * a.H + item_i) * C + sub * V);
#pragma unroll
        for (int x = 0; x < V; x += 4) {
          const float4 q4 = __ldg(reinterpret_cast<const float4 *>(gp + x));
          go[x] = q4.x; go[x + 1] = q4.y; go[x + 2] = q4.z; go[x + 3] = q4.w;
        }
      } else {
#pragma unroll
        for (int x = 0; x < V; ++x) go[x] = 0.f;
      }
#pragma unroll 1
      for (int r0 = 0; r0 < nrows; r0 += GPI * U) {
        RowEntry e[U];
        float v[U][V];
#pragma unroll
        for (int u = 0; u < U; ++u) e[u] = table[base + r0 + u];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (e[u].off >= 0) {
            RowVec4<VT>::load(vbase + e[u].off, v[u]);
          } else {
#pragma unroll
            for (int x = 0; x < V; ++x) v[u][x] = 0.f;
          }
        }
        float d[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          d[u] = 0.f;
#pragma unroll
          for (int x = 0; x < V; ++x) d[u] = fmaf(v[u][x], go[x], d[u]);
        }
        int u_mine;
        const float f = fold_four_dots<G>(d, sub, u_mine);
        if (u_mine >= 0) dot_slots[base + r0 + u_mine] = f;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (e[u].off >= 0 && e[u].wgt != 0.f) {
            float *gp = gvbase + e[u].off;
#pragma unroll
            for (int x = 0; x < V; x += 4)
              red_add_v4(gp + x, e[u].wgt * go[x], e[u].wgt * go[x + 1], e[u].wgt * go[x + 2],
                         e[u].wgt * go[x + 3]);
          }
        }
      }
    }
    __syncwarp();
    const float4 tq = reinterpret_cast<const float4 *>(dot_slots)[lane];
    const float tt[4] = {tq.x, tq.y, tq.z, tq.w};
    float part = bwd_point_epilogue<DT, MODE>(a, c, j, st, tt);
    if (mode_from_offsets(MODE)) {
      // softmax backward, grad_logit_j = a_j * (g_j - sum_k a_k g_k): the sum runs over the softmax's lanes; g_j was
      // parked in grad_attn by the epilogue.  2-D: the weight in hand is a_j / maps.
      for (int s = lanes / 2; s > 0; s >>= 1) part += __shfl_xor_sync(0xffffffffu, part, s);
      if (MODE == kCallerFused2D) part *= (float)a.maps;
      if (live) {
        float *g = a.grad_attn + (c.attn - a.attn) + j;
        *g = st.aw * (*g - part);
      }
    }
    __syncwarp();
  }
}

// ------------------------------------------------------------------------------------------------
// host-side dispatch
// ------------------------------------------------------------------------------------------------
template <typename VT, typename DT, int C, int MODE, int LPP>
void launch_k(KArgs &a, int cams, cudaStream_t s) {
  constexpr auto kernel = dfa3d_backward_packed_kernel<VT, DT, C, MODE, LPP>;
  constexpr unsigned kBatch = kWarpsPerCta * (32 / LPP);             // items a CTA takes at a time
  const unsigned batches = ((unsigned)a.items_per_cam + kBatch - 1) / kBatch;
  a.rounds = walk_backward(batches, cams, kPackedRounds, resident_ctas<kernel>(), sm_count());
  kernel<<<dim3((batches + a.rounds - 1) / a.rounds, (unsigned)cams, 1), kThreads, 0, s>>>(a);
}

template <typename VT, typename DT, int MODE, int LPP>
void launch_c(KArgs &a, int cams, cudaStream_t s) {
  if (a.C == 16) launch_k<VT, DT, 16, MODE, LPP>(a, cams, s);
  else if (a.C == 32) launch_k<VT, DT, 32, MODE, LPP>(a, cams, s);
  else launch_k<VT, DT, 64, MODE, LPP>(a, cams, s);
}

template <typename VT, typename DT, int MODE>
cudaError_t launch_vd(const KArgs &a0, cudaStream_t s) {
  // (2-D from offsets: the kernels are made for the lanes of a map)
  const int lpp = MODE == kCallerFused2D ? lanes_of_points(a0.LP)
                                         : packed_lanes(a0.LP, a0.C, RowVec4<VT>::kElems, a0.items, true, mode_has_depth(MODE),
                                                        sm_count());
  for (int b0 = 0; b0 < a0.B; b0 += 65535) {      // grid.y limit
    KArgs a = a0;
    a.b0 = b0;
    const int cams = min(65535, a0.B - b0);
    if (lpp == 4) launch_c<VT, DT, MODE, 4>(a, cams, s);
    else if (lpp == 8) launch_c<VT, DT, MODE, 8>(a, cams, s);
    else launch_c<VT, DT, MODE, 16>(a, cams, s);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

template <int MODE>
cudaError_t launch_m(const KArgs &a, int value_dtype, int dist_dtype, cudaStream_t s) {
  if (value_dtype == kDtypeF16) return launch_vd<__half, __half, MODE>(a, s);
  if (value_dtype == kDtypeBF16)
    return dist_dtype == kDtypeBF16 ? launch_vd<__nv_bfloat16, __nv_bfloat16, MODE>(a, s)
                                    : launch_vd<__nv_bfloat16, float, MODE>(a, s);
  return dist_dtype == kDtypeBF16 ? launch_vd<float, __nv_bfloat16, MODE>(a, s) : launch_vd<float, float, MODE>(a, s);
}

}  // namespace

cudaError_t launch_backward_packed(const KArgs &a, int value_dtype, int dist_dtype, int mode, cudaStream_t s) {
  if (mode == kCallerFused2D)
    return value_dtype == kDtypeF32 ? launch_vd<float, float, kCallerFused2D>(a, s) : cudaErrorNotSupported;
  if (mode == kGivenDepthScore) {
    if (value_dtype == kDtypeF16) return launch_vd<__half, float, kGivenDepthScore>(a, s);
    return value_dtype == kDtypeBF16 ? launch_vd<__nv_bfloat16, float, kGivenDepthScore>(a, s)
                                     : launch_vd<float, float, kGivenDepthScore>(a, s);
  }
  if (mode == kCallerFused) return launch_m<kCallerFused>(a, value_dtype, dist_dtype, s);
  return launch_m<kFused>(a, value_dtype, dist_dtype, s);
}

}  // namespace dfa3d
