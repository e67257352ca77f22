// DFA3D forward kernels (sm_100a).
//
// One warp owns one (camera b, query q, head h) item.  The L*P sampling points of the item are taken
// 32 at a time:
//   prologue  -- lane j owns point j: it reads its location and attention weight (coalesced), derives
//                the four bilinear corners, and (fused mode) gathers the 8 depth-distribution values
//                that give the four per-corner depth scores; it leaves one {row offset, weight} pair
//                per corner in the warp's slice of shared memory;
//   gather    -- the warp walks the (point, corner) rows; a group of G lanes reads one value row with
//                16-byte loads (4 fp32 or 8 bf16 channels per lane), so one warp-wide request fetches
//                32/G rows, and every lane
//                accumulates weight * row fragment;
//   epilogue  -- the 32/G partial sums are folded with xor-shuffles and the output row is stored.
// This replaces the reference's pair of kernels (one thread per (b,q,h) for the depth scores,
// ms_depth_score_sample_cuda_kernel.cuh:94-148; one thread per output channel for the attention,
// wms_deform_attn_cuda_kernel.cuh:240-303) and the depth_score round trip through HBM between them.
//
// The kernels are issue-bound as much as memory-bound (ncu: issue slots 2/3 busy), so index
// arithmetic is kept 32-bit: the grid's y dimension is the camera, 64-bit bases are formed once per
// warp, and when L*P is a multiple of 32 (FULL) the row loop has a compile-time trip count.
#include "dfa3d_forward_point.cuh"
#include "dfa3d_launch.h"

namespace dfa3d {

// ------------------------------------------------------------------------------------------------
// fused / given-depth-score / caller-fused forward; C/V a power of two, V = channels per 16 bytes
// ------------------------------------------------------------------------------------------------
// One item: the L*P points of (camera c.b, query, head c.h), 32 at a time; `table` is the warp's slice
// of the row table in shared memory.
template <typename VT, typename DT, int C, int MODE, bool WRITE_DS, bool FULL>
__device__ __forceinline__ void forward_item(const KArgs &a, const LevelTable &lv, const ItemCtx &c,
                                             RowTable &table, int lane) {
  constexpr int V = RowVec<VT>::kElems;   // channels per lane
  constexpr int G = C / V;                // lanes per row
  constexpr int R = 32 / G;               // rows per warp-wide request
  constexpr int U = 4;                    // requests in flight per lane: the corners of a group's point
  static_assert(G >= 1 && G <= 32 && (G & (G - 1)) == 0, "C/V must be a power of two <= 32");
  const VT *vbase = reinterpret_cast<const VT *>(a.value) + (((long long)c.b * a.N * a.H + c.h) * C +
                                                             (lane % G) * V);

  float acc[V];
#pragma unroll
  for (int i = 0; i < V; ++i) acc[i] = 0.f;
  SoftmaxStats sm{0.f, 1.f};
  if (MODE == kCallerFused) sm = item_softmax_stats(a, c, lane);

  for (int chunk = 0; chunk < a.LP; chunk += 32) {
    float ds[4], wgt[4];
    int off[4];
    fwd_point<DT, MODE>(a, lv, c, chunk + lane, sm, ds, wgt, off);
    table.store(lane, off, wgt);
    if (WRITE_DS && chunk + lane < a.LP)
      reinterpret_cast<float4 *>(a.ds_out)[c.pt0 + chunk + lane] = make_float4(ds[0], ds[1], ds[2], ds[3]);
    __syncwarp();
    // R points per step: U independent row-fragment loads in flight per lane, then U fused multiply-adds.
    auto step = [&](int p0) {
      RowEntry e[U];
      float v[U][V];
      table.load(p0 + lane / G, e);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (e[u].off >= 0) {
          RowVec<VT>::load(vbase + e[u].off, v[u]);
        } else {
#pragma unroll
          for (int i = 0; i < V; ++i) v[u][i] = 0.f;
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int i = 0; i < V; ++i) acc[i] = fmaf(e[u].wgt, v[u][i], acc[i]);
    };
    if constexpr (FULL && V == 8) {
      // 16-bit rows stay packed until they are summed, so that a lane's next row can be asked for as soon as the last one in
      // its place is used up: bf16, 6 cameras of the base levels, uniform locations 504 -> 491 us, fp16 with depth scores
      // 288 -> 275 (fp32 rows, which take as many registers packed or not: no gain)
      RowEntry e[U], next[U];
      uint4 v[U];
      auto fetch = [&](int off, uint4 &r) {
        r = make_uint4(0, 0, 0, 0);
        if (off >= 0) r = __ldg(reinterpret_cast<const uint4 *>(vbase + off));
      };
      table.load(lane / G, e);
#pragma unroll
      for (int u = 0; u < U; ++u) fetch(e[u].off, v[u]);
#pragma unroll
      for (int p0 = 0; p0 < 32; p0 += R) {
        const bool more = p0 + R < 32;
        if (more) table.load(p0 + R + lane / G, next);
#pragma unroll
        for (int u = 0; u < U; ++u) {
          float t[V];
          RowVec<VT>::widen(v[u], t);
#pragma unroll
          for (int i = 0; i < V; ++i) acc[i] = fmaf(e[u].wgt, t[i], acc[i]);
          if (more) {
            fetch(next[u].off, v[u]);
            e[u] = next[u];
          }
        }
      }
    } else if constexpr (FULL) {          // compile-time trip count, table offsets become immediates
#pragma unroll
      for (int p0 = 0; p0 < 32; p0 += R) step(p0);
    } else {
      const int n = min(32, a.LP - chunk);         // (the table's slots past the last point hold no rows)
#pragma unroll 1
      for (int p0 = 0; p0 < n; p0 += R) step(p0);
    }
    __syncwarp();
  }
  fold_and_store<V, G, R>(acc, lane, a.out + (c.item * C + lane % G * V), true);
}

// 5 CTAs (40 warps) per SM: measured best; at 6+ the register cap starts to cost more than the
// extra warps hide.  A CTA walks up to DFA3D_FWD_ITEMS_PER_WARP consecutive groups of 8 items (the grid's
// ~60 000 CTAs per camera otherwise live ~2 us each and their turnover shows: measured -7 % at 8).
// WALK: that number, as every launch of some size has it; 0: a.rounds of them (dfa3d_walk.h).  As a run-time number it costs
// registers that most kernels do not have: 6 cameras of the base levels, us at run time / as a constant: bf16 of 32 channels
// 524 / 519, of 64 from offsets 503 / 491, fp32 of 64 535 / 521, fp16 of 20 points 363 / 350.  Unrolled, fp32 rows of up to 32
// channels were faster with the run-time number (base 565 / 569, 8 channels from offsets 348 / 371, bf16 dist from offsets
// 435 / 459), as were bf16 rows of 32 with fp32 dist (6000 queries 330 / 341).
template <typename VT, typename DT, int C, int MODE, bool WRITE_DS, bool FULL, int WALK>
__global__ void __launch_bounds__(kThreads, DFA3D_FWD_MIN_CTAS)
dfa3d_forward_kernel(const KArgs a) {
  __shared__ LevelTable lv;
  __shared__ RowTable rows[kWarpsPerCta];
  stage_levels(lv, a);
  const int rounds = WALK ? WALK : a.rounds;
  if (MODE == kCallerFused) {
    const unsigned items = kWarpsPerCta * (unsigned)rounds;
    prefetch_offsets(a, (int)blockIdx.y + a.b0, blockIdx.x * items, items);
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll 1
  for (int it = 0; it < rounds; ++it) {
    ItemCtx c;
    if (!item_context<MODE, DFA3D_FWD_HEAD_MAJOR != 0>(a, warp, blockIdx.x * rounds + it, c)) return;
    forward_item<VT, DT, C, MODE, WRITE_DS, FULL>(a, lv, c, rows[warp], lane);
  }
}

// ------------------------------------------------------------------------------------------------
// any C: lanes stride over channels, rows walked one by one (correctness path for unusual widths)
// ------------------------------------------------------------------------------------------------
template <typename VT, typename DT, int MODE, bool WRITE_DS>
__global__ void __launch_bounds__(kThreads)
dfa3d_forward_generic_kernel(const KArgs a) {
  __shared__ LevelTable lv;
  __shared__ __align__(16) RowEntry rows[kWarpsPerCta][128];
  stage_levels(lv, a);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  ItemCtx c;
  if (!item_context<MODE>(a, warp, blockIdx.x, c)) return;
  const int C = a.C;
  const VT *vbase = reinterpret_cast<const VT *>(a.value) + ((long long)c.b * a.N * a.H + c.h) * C;
  RowEntry *my = rows[warp];
  SoftmaxStats sm{0.f, 1.f};
  if (MODE == kCallerFused) sm = item_softmax_stats(a, c, lane);
  for (int c0 = 0; c0 < C; c0 += 32) {          // C <= 1024: at most 32 passes
    const int ch = c0 + lane;
    float acc = 0.f;
    for (int chunk = 0; chunk < a.LP; chunk += 32) {
      float ds[4], wgt[4];
      int off[4];
      fwd_point<DT, MODE>(a, lv, c, chunk + lane, sm, ds, wgt, off);
      store_rows(my, lane, off, wgt);
      if (WRITE_DS && c0 == 0 && chunk + lane < a.LP)
        reinterpret_cast<float4 *>(a.ds_out)[c.pt0 + chunk + lane] =
            make_float4(ds[0], ds[1], ds[2], ds[3]);
      __syncwarp();
      const int nrows = min(32, a.LP - chunk) * 4;
      if (ch < C)
        for (int r = 0; r < nrows; ++r) {
          const RowEntry e = my[r];
          if (e.off >= 0) acc = fmaf(e.wgt, load_scalar(vbase + e.off + ch), acc);
        }
      __syncwarp();
    }
    if (ch < C) a.out[c.item * C + ch] = acc;
  }
}

// ------------------------------------------------------------------------------------------------
// depth scores only (two-stage API): one thread per sampling point
// ------------------------------------------------------------------------------------------------
template <typename DT>
__global__ void __launch_bounds__(kThreads)
dfa3d_depth_score_forward_kernel(const KArgs a) {
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
    const DT *dist_bh = reinterpret_cast<const DT *>(a.dist) +
                        ((long long)b * a.Nd * a.dist_pix_stride + h * a.dist_head_stride);
    float ds[4];
    const float hd = 1.f - g.ld;
    const int Dlim = min(g.Dd, a.D);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float lo, hi;
      load_depth_pair(dist_bh, a.dist_pix_stride, g.dpix[k], g.z0, Dlim, g.ok3, lo, hi);
      ds[k] = g.ok3 ? lo * hd + hi * g.ld : 0.f;
    }
    reinterpret_cast<float4 *>(a.ds_out)[pt] = make_float4(ds[0], ds[1], ds[2], ds[3]);
  }
}

// ------------------------------------------------------------------------------------------------
// host-side dispatch
// ------------------------------------------------------------------------------------------------
static dim3 item_grid(const KArgs &a, int cams, int items_per_warp) {
  const int per_cta = kWarpsPerCta * items_per_warp;
  return dim3((unsigned)((a.items_per_cam + per_cta - 1) / per_cta), (unsigned)cams, 1);
}

template <typename VT, typename DT, int C, int MODE, bool WRITE_DS, bool FULL>
static void launch_forward_c(KArgs &a, int cams, cudaStream_t s) {
  // unrolled, fp32 rows of up to 32 channels or bf16 rows of 32 with fp32 dist: one kernel for every launch (see the kernel)
  constexpr bool kOne = FULL && (RowVec<VT>::kElems == 4 ? C <= 32 : C == 32 && MODE == kFused && sizeof(DT) == 4 && !WRITE_DS);
  constexpr int kMost = DFA3D_FWD_ITEMS_PER_WARP;
  constexpr auto kLong = dfa3d_forward_kernel<VT, DT, C, MODE, WRITE_DS, FULL, kOne ? 0 : kMost>;
  constexpr auto kShort = dfa3d_forward_kernel<VT, DT, C, MODE, WRITE_DS, FULL, 0>;
  // a group of 32 points is long beside the start of a CTA; a chain of loads weighs as much as a resident CTA's share
  a.rounds = walk_forward((a.items_per_cam + kWarpsPerCta - 1) / kWarpsPerCta, cams, kMost, resident_ctas<kLong>(), sm_count(),
                          WalkCost{2, 8});
  const dim3 grid = item_grid(a, cams, a.rounds);
  if (a.rounds == kMost) kLong<<<grid, kThreads, 0, s>>>(a);
  else kShort<<<grid, kThreads, 0, s>>>(a);
}

template <typename VT, typename DT, int MODE, bool WRITE_DS, bool FULL>
static void launch_forward_g(KArgs &a, int cams, cudaStream_t s) {
  constexpr int V = RowVec<VT>::kElems;
  switch ((a.C % V == 0) ? a.C / V : 0) {
    case 2:  launch_forward_c<VT, DT, 2 * V, MODE, WRITE_DS, FULL>(a, cams, s); break;
    case 4:  launch_forward_c<VT, DT, 4 * V, MODE, WRITE_DS, FULL>(a, cams, s); break;
    case 8:  launch_forward_c<VT, DT, 8 * V, MODE, WRITE_DS, FULL>(a, cams, s); break;
    case 16: launch_forward_c<VT, DT, 16 * V, MODE, WRITE_DS, FULL>(a, cams, s); break;
    case 32: launch_forward_c<VT, DT, 32 * V, MODE, WRITE_DS, FULL>(a, cams, s); break;
    default:
      dfa3d_forward_generic_kernel<VT, DT, MODE, WRITE_DS><<<item_grid(a, cams, 1), kThreads, 0, s>>>(a);
      break;
  }
}

template <typename VT, typename DT, int MODE, bool WRITE_DS>
static void launch_forward_ds(KArgs &a, int cams, cudaStream_t s) {
  if (a.LP % 32 == 0) launch_forward_g<VT, DT, MODE, WRITE_DS, true>(a, cams, s);
  else launch_forward_g<VT, DT, MODE, WRITE_DS, false>(a, cams, s);
}

template <typename VT, typename DT, int MODE>
static cudaError_t launch_forward_vd(const KArgs &a0, cudaStream_t s) {
  for (int b0 = 0; b0 < a0.B; b0 += 65535) {      // grid.y limit
    KArgs a = a0;
    a.b0 = b0;
    const int cams = min(65535, a0.B - b0);
    if constexpr (MODE == kFused) {               // the other modes' entry points return no depth score
      if (a.ds_out) launch_forward_ds<VT, DT, MODE, true>(a, cams, s);
      else launch_forward_ds<VT, DT, MODE, false>(a, cams, s);
    } else {
      launch_forward_ds<VT, DT, MODE, false>(a, cams, s);
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// Storage types are the DFA3D_DTYPE_* codes of the C header.  fp32 and bf16 combine freely; fp16 value
// goes with fp16 dist (what a half-precision caller passes) -- the C entry points reject the rest.
template <int MODE>
static cudaError_t launch_forward_m(const KArgs &a, int value_dtype, int dist_dtype, cudaStream_t s) {
  if (value_dtype == kDtypeF16) return launch_forward_vd<__half, __half, MODE>(a, s);
  if (value_dtype == kDtypeBF16)
    return dist_dtype == kDtypeBF16 ? launch_forward_vd<__nv_bfloat16, __nv_bfloat16, MODE>(a, s)
                                    : launch_forward_vd<__nv_bfloat16, float, MODE>(a, s);
  return dist_dtype == kDtypeBF16 ? launch_forward_vd<float, __nv_bfloat16, MODE>(a, s)
                                  : launch_forward_vd<float, float, MODE>(a, s);
}

cudaError_t launch_forward(const KArgs &a, int value_dtype, int dist_dtype, int mode, cudaStream_t s) {
  if (a.items == 0) return cudaSuccess;
  if (packed_covers(a.LP, a.C)) return launch_forward_packed(a, value_dtype, dist_dtype, mode, s);
  if (mode == kCallerFused2D) return cudaErrorNotSupported;       // see attn2d_supported
  if (mode == kGivenDepthScore) {   // dist is not read: its type parameter is irrelevant
    if (value_dtype == kDtypeF16) return launch_forward_vd<__half, float, kGivenDepthScore>(a, s);
    return value_dtype == kDtypeBF16 ? launch_forward_vd<__nv_bfloat16, float, kGivenDepthScore>(a, s)
                                     : launch_forward_vd<float, float, kGivenDepthScore>(a, s);
  }
  if (mode == kCallerFused) return launch_forward_m<kCallerFused>(a, value_dtype, dist_dtype, s);
  return launch_forward_m<kFused>(a, value_dtype, dist_dtype, s);
}

cudaError_t launch_depth_score_forward(const KArgs &a, int dist_dtype, cudaStream_t s) {
  const long long npts = a.items * a.LP;
  if (npts == 0) return cudaSuccess;
  const unsigned grid = (unsigned)min((npts + kThreads - 1) / kThreads, (long long)148 * 64);
  if (dist_dtype == kDtypeF16) dfa3d_depth_score_forward_kernel<__half><<<grid, kThreads, 0, s>>>(a);
  else if (dist_dtype == kDtypeBF16) dfa3d_depth_score_forward_kernel<__nv_bfloat16><<<grid, kThreads, 0, s>>>(a);
  else dfa3d_depth_score_forward_kernel<float><<<grid, kThreads, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace dfa3d
