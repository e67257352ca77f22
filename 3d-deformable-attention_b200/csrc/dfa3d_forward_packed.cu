// DFA3D forward for items of few points (L*P <= 16): a warp takes several consecutive items at once (sm_100a).
//
// With one item per warp an item of 4 points (temporal self-attention and the decoder's cross-attention
// use 1 level x 4 points) keeps 4 lanes busy in the prologue and costs a whole chain of dependent
// latencies (locations -> row table -> rows -> sum -> store) for 16 rows.  Here an item has LPP lanes -- 4, 8 or 16
// (packed_lanes) -- and lane j of them owns its point j, so the prologue is (nearly) full and coalesced:
// the points of consecutive items are consecutive in memory.  A group of G lanes then sums all rows of one item (or,
// when the warp holds fewer items than groups, a share of them) and writes that item's output itself.
// Bound like the one-item kernels by the rows that travel from L2 to the SM.  Against one item per warp, 6 cameras x 6000
// queries x 8 heads of fp32: 3 levels x 4 points of 32 channels 205 -> 142 us, 1 x 5 points of 16 channels 150 -> 64 us.
#include "dfa3d_forward_point.cuh"
#include "dfa3d_launch.h"

namespace dfa3d {
namespace {

// CTAs per SM the kernel is compiled for.  fp32 rows: 6 (48 warps; the kernel waits on chains of dependent loads)
// measured 1-4 % faster than 5 and 4-8 % faster than 4 -- but not where the depth scores are kept to be written: the
// 40 registers then spill up to 270 bytes (1 level x 8 points, 6 x 6000 queries: 142 us at 6).  16-bit rows hold eight
// channels a lane.
template <typename VT, int MODE, bool WRITE_DS>
struct PackedCtas { static constexpr int value = RowVec<VT>::kElems == 8 ? 4 : WRITE_DS ? 5 : 6; };

// EXACT: L*P == LPP, the row loop is unrolled; otherwise it ends at the item's last row.
// TURNS: an item that a small launch gives more lanes than its points need (packed_lanes) has TURNS times the groups.  They
// read their rows at the same time, but add them up one after the other, in the order in which the fewer groups of another
// launch do: an item's result does not depend on what else the launch holds.
template <typename VT, typename DT, int C, int MODE, bool WRITE_DS, int LPP, bool EXACT, int TURNS>
__global__ void __launch_bounds__(kThreads, PackedCtas<VT, MODE, WRITE_DS>::value)
dfa3d_forward_packed_kernel(const KArgs a) {
  constexpr int V = RowVec<VT>::kElems;
  constexpr int G = C / V;                      // lanes per row
  constexpr int R = 32 / G;                     // groups per warp
  constexpr int K = 32 / LPP;                   // items per warp
  constexpr int GPI = R > K ? R / K : 1;        // groups sharing one item
  constexpr int IPG = K > R ? K / R : 1;        // items one group handles in turn
  constexpr int U = 4;
  // Fully unrolled is 1-8 % faster than by 2 -- except where a group has one item of its own and no dist to wait for: the
  // loads of the whole item are then moved to the front and spill 170 to 240 bytes (1 level x 8 points, 6 x 6000
  // queries: 122 us fully unrolled, 75 by 2; 2-D from offsets, 22500 queries: 88, 63 by 2, 62 by 4).
  constexpr bool kShort = !mode_has_depth(MODE) && GPI == 1 && IPG == 1;
  constexpr int kUnroll = !kShort ? LPP / GPI : MODE == kCallerFused2D ? 4 : 2;
  // fold_and_store where there is something to halve (16-bit rows whose item is shared), and for fp32 rows where the kernel is
  // faster with it: rows in a loop that is not unrolled, no scores (us without / with: 5 points of 64 channels, 6 x 6000
  // queries 113.7 / 106.9, 10 of 32 in 2-D, 3 x 6000 57.6 / 54.9, 900 queries of 8 in 16 lanes 9.3 / 7.7, bf16 dist from
  // offsets 68.5 / 66.5); 2-D from offsets, 900 x 16 points 8.80 / 8.61; 16 points of 32 channels without scores (6 x 6000
  // queries, 2-D 126.3 / 124.1, with two levels 139.5 / 136.8, from offsets 174.7 / 173.4; of 16 channels 109.2 / 110.5).  It cost
  // the others registers: 2-D from offsets, 40000 queries x 4 points 51.8 / 53.8; 16 points of 16 channels with scores 165.8 /
  // 173.3; fp16, 8 points of 64 channels 126 / 133.
  constexpr bool kFold = V == 8 || MODE == kCallerFused2D ? GPI / TURNS > 1 : !WRITE_DS && (!EXACT || (GPI == 2 && C == 32));
  constexpr int SUMS = GPI / TURNS;             // partial sums of an item
  static_assert(32 % LPP == 0 && 32 % G == 0 && LPP % GPI == 0, "unsupported packing");
  static_assert(GPI % TURNS == 0 && (TURNS == 1 || (!EXACT && IPG == 1)), "unsupported packing");
  __shared__ LevelTable lv;
  __shared__ RowTable rows[kWarpsPerCta];
  stage_levels(lv, a);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane % G, grp = lane / G;
  const int b = (int)blockIdx.y + a.b0;
  const VT *vbase = reinterpret_cast<const VT *>(a.value) + ((long long)b * a.N * a.H * C + sub * V);
  RowTable &table = rows[warp];
  // the camera's queries: rows [q0, q0 + nq) of the per-query tensors
  const long long q0 = a.q_off ? (long long)__ldg(a.q_off + b) : (long long)b * a.Q;
  const unsigned nitems = (unsigned)(a.q_off ? __ldg(a.q_off + b + 1) - (int)q0 : a.Q) * (unsigned)a.H;
  const int n = EXACT ? LPP : a.LP;
#pragma unroll 1
  for (int it = 0; it < a.rounds; ++it) {
    const unsigned first = ((blockIdx.x * a.rounds + it) * kWarpsPerCta + warp) * K;
    if (first >= nitems) return;
    {
      const unsigned idx = first + lane / LPP;
      const int j = lane % LPP;
      const bool live = idx < nitems && (EXACT || j < a.LP);
      ItemCtx c;
      c.b = b;
      const unsigned inside = min(idx, nitems - 1);           // (past the end: the last item, which is there to read)
      const unsigned q = inside / (unsigned)a.H;
      c.h = (int)(inside - q * (unsigned)a.H);
      c.bq = q0 + q;
      c.item = q0 * a.H + inside;
      item_inputs<MODE>(a, c);
      SoftmaxStats sm{0.f, 1.f};
      if (mode_from_offsets(MODE))
        sm = lanes_softmax_stats(live ? __ldg(c.attn + j) : 0.f, live, MODE == kCallerFused2D ? LPP / a.maps : LPP);
      float ds[4], wgt[4];
      int off[4];
      fwd_point<DT, MODE>(a, lv, c, live ? j : a.LP, sm, ds, wgt, off);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (off[k] >= 0) off[k] += c.h * C;     // rows of different heads share the table
      table.store(lane, off, wgt);
      if (WRITE_DS && live)
        reinterpret_cast<float4 *>(a.ds_out)[c.pt0 + j] = make_float4(ds[0], ds[1], ds[2], ds[3]);
    }
    __syncwarp();
#pragma unroll 1                               // unrolled too, 4 points an item spilled 70 to 140 bytes
    for (int t = 0; t < IPG; ++t) {
      const int i = grp / GPI + t * (R / GPI);  // item of the warp this group works on
      const int base = i * LPP + grp % GPI;     // its first point
      float acc[V];
#pragma unroll
      for (int x = 0; x < V; ++x) acc[x] = 0.f;
      auto step = [&](int p0) {
        RowEntry e[U];
        float v[U][V];
        table.load(base + p0, e);
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (e[u].off >= 0) {
            RowVec<VT>::load(vbase + e[u].off, v[u]);
          } else {
#pragma unroll
            for (int x = 0; x < V; ++x) v[u][x] = 0.f;
          }
        }
#pragma unroll
        for (int turn = 0; turn < TURNS; ++turn) {
#pragma unroll
          for (int u = 0; u < U; ++u)
#pragma unroll
            for (int x = 0; x < V; ++x) acc[x] = fmaf(e[u].wgt, v[u][x], acc[x]);
          if (TURNS > 1) {                     // all go on from the sum of the group whose turn it was
#pragma unroll
            for (int x = 0; x < V; ++x)
              acc[x] = __shfl_sync(0xffffffffu, acc[x], (grp / GPI * GPI + turn * SUMS + grp % SUMS) * G + sub);
          }
        }
      };
      if (EXACT) {
#pragma unroll kUnroll
        for (int p0 = 0; p0 < LPP; p0 += GPI) step(p0);
      } else {
#pragma unroll 1
        for (int p0 = 0; p0 < n; p0 += GPI) step(p0);     // (past the last point the table holds no rows)
      }
      const unsigned idx = first + i;
      if constexpr (kFold) {
        fold_and_store<V, G, SUMS>(acc, lane, a.out + ((q0 * a.H + idx) * C + sub * V), idx < nitems && grp % GPI < SUMS);
      } else {
#pragma unroll
        for (int s = G; s < G * SUMS; s <<= 1)
#pragma unroll
          for (int x = 0; x < V; ++x) acc[x] += __shfl_xor_sync(0xffffffffu, acc[x], s);
        if (grp % GPI == 0 && idx < nitems) {
          float *o = a.out + ((q0 * a.H + idx) * C + sub * V);
#pragma unroll
          for (int x = 0; x < V; x += 4)
            *reinterpret_cast<float4 *>(o + x) = make_float4(acc[x], acc[x + 1], acc[x + 2], acc[x + 3]);
        }
      }
    }
    __syncwarp();
  }
}

// ------------------------------------------------------------------------------------------------
// host-side dispatch
// ------------------------------------------------------------------------------------------------
template <typename VT, typename DT, int C, int MODE, bool WRITE_DS, int LPP, bool EXACT, int LANES>
void launch_k(KArgs &a, int cams, cudaStream_t s) {
  constexpr int V = RowVec<VT>::kElems, kTurns = groups_of_item(C, V, LPP) / groups_of_item(C, V, LANES);
  constexpr auto kernel = dfa3d_forward_packed_kernel<VT, DT, C, MODE, WRITE_DS, LPP, EXACT, kTurns>;
  constexpr unsigned kBatch = kWarpsPerCta * (32 / LPP);             // items a CTA takes at a time
  const unsigned batches = ((unsigned)a.items_per_cam + kBatch - 1) / kBatch;
  // unrolled, a batch takes nearly as long alone as beside others, and a CTA's start counts more
  a.rounds = walk_forward(batches, cams, kPackedRounds, resident_ctas<kernel>(), sm_count(), EXACT ? WalkCost{8, 24} : WalkCost{6, 8});
  kernel<<<dim3((batches + a.rounds - 1) / a.rounds, (unsigned)cams, 1), kThreads, 0, s>>>(a);
}

// LANES: what the item's points need, LPP: what it gets
template <typename VT, typename DT, int MODE, bool WRITE_DS, int LPP, bool EXACT, int LANES = LPP>
void launch_c(KArgs &a, int cams, cudaStream_t s) {
  if (a.C == 16) launch_k<VT, DT, 16, MODE, WRITE_DS, LPP, EXACT, LANES>(a, cams, s);
  else if (a.C == 32) launch_k<VT, DT, 32, MODE, WRITE_DS, LPP, EXACT, LANES>(a, cams, s);
  else launch_k<VT, DT, 64, MODE, WRITE_DS, LPP, EXACT, LANES>(a, cams, s);
}

template <typename VT, typename DT, int MODE, bool WRITE_DS>
void launch_lp(KArgs &a, int lpp, int cams, cudaStream_t s) {
  // the unrolled loop is instantiated where it is the common case: fp32 throughout
  constexpr bool kFloat = sizeof(VT) == 4 && (sizeof(DT) == 4 || !mode_has_depth(MODE));
  if constexpr (kFloat) {
    if (a.LP == lpp) {
      if (lpp == 4) launch_c<VT, DT, MODE, WRITE_DS, 4, true>(a, cams, s);
      else if (lpp == 8) launch_c<VT, DT, MODE, WRITE_DS, 8, true>(a, cams, s);
      else launch_c<VT, DT, MODE, WRITE_DS, 16, true>(a, cams, s);
      return;
    }
  }
  if constexpr (MODE != kCallerFused2D) {      // attn2d_supported: fp32, exact
    if (lpp == 4) launch_c<VT, DT, MODE, WRITE_DS, 4, false>(a, cams, s);
    else if (lpp == 8) {
      if (a.LP <= 4) launch_c<VT, DT, MODE, WRITE_DS, 8, false, 4>(a, cams, s);
      else launch_c<VT, DT, MODE, WRITE_DS, 8, false>(a, cams, s);
    } else {
      if (a.LP <= 4) launch_c<VT, DT, MODE, WRITE_DS, 16, false, 4>(a, cams, s);
      else if (a.LP <= 8) launch_c<VT, DT, MODE, WRITE_DS, 16, false, 8>(a, cams, s);
      else launch_c<VT, DT, MODE, WRITE_DS, 16, false>(a, cams, s);
    }
  }
}

template <typename VT, typename DT, int MODE>
cudaError_t launch_vd(const KArgs &a0, cudaStream_t s) {
  // (2-D from offsets: the kernels are made for the lanes of a map)
  const int lpp = MODE == kCallerFused2D ? lanes_of_points(a0.LP)
                                         : packed_lanes(a0.LP, a0.C, RowVec<VT>::kElems, a0.items, false, mode_has_depth(MODE),
                                                        sm_count());
  for (int b0 = 0; b0 < a0.B; b0 += 65535) {      // grid.y limit
    KArgs a = a0;
    a.b0 = b0;
    const int cams = min(65535, a0.B - b0);
    if constexpr (mode_from_offsets(MODE)) {      // the caller-fused entry points return no depth score
      launch_lp<VT, DT, MODE, false>(a, lpp, cams, s);
    } else if constexpr (MODE == kFused) {
      if (a.ds_out) launch_lp<VT, DT, MODE, true>(a, lpp, cams, s);
      else launch_lp<VT, DT, MODE, false>(a, lpp, cams, s);
    } else {
      launch_lp<VT, DT, MODE, false>(a, lpp, cams, s);
    }
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

cudaError_t launch_forward_packed(const KArgs &a, int value_dtype, int dist_dtype, int mode, cudaStream_t s) {
  if (mode == kCallerFused2D)
    return value_dtype == kDtypeF32 ? launch_vd<float, float, kCallerFused2D>(a, s) : cudaErrorNotSupported;
  if (mode == kGivenDepthScore) {   // dist is not read: its type parameter is irrelevant
    if (value_dtype == kDtypeF16) return launch_vd<__half, float, kGivenDepthScore>(a, s);
    return value_dtype == kDtypeBF16 ? launch_vd<__nv_bfloat16, float, kGivenDepthScore>(a, s)
                                     : launch_vd<float, float, kGivenDepthScore>(a, s);
  }
  if (mode == kCallerFused) return launch_m<kCallerFused>(a, value_dtype, dist_dtype, s);
  return launch_m<kFused>(a, value_dtype, dist_dtype, s);
}

}  // namespace dfa3d
