// Forward of one sampling point: shared by the kernels with one item per warp and with several.
#pragma once
#include "dfa3d_common.cuh"

namespace dfa3d {

// ------------------------------------------------------------------------------------------------
// prologue: per-lane point -> 4 row entries (+ depth scores)
// ------------------------------------------------------------------------------------------------
template <typename DT, int MODE>
__device__ __forceinline__ void fwd_point(const KArgs &a, const LevelTable &lv, const ItemCtx &c, int j,
                                          const SoftmaxStats &sm, float (&ds)[4], float (&wgt)[4],
                                          int (&off)[4]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) { ds[k] = 0.f; wgt[k] = 0.f; off[k] = -1; }
  if (j >= a.LP) return;
  const int l = j / a.P;
  float x, y, z, aw;
  read_point<MODE>(a, lv, c, j, l, sm, x, y, z, aw);
  const PointGeo g = point_geometry(x, y, z, mode_has_depth(MODE), lv.h[l], lv.w[l], lv.d[l], lv.start[l],
                                    a.N, dist_map_of(a, lv, l));
  if (!g.ok2) return;
  float bw[4];
  bilinear_weights(g, bw);
  if (mode_has_depth(MODE)) {
    const DT *dist_bh = reinterpret_cast<const DT *>(a.dist) +
                        ((long long)c.b * a.Nd * a.dist_pix_stride + c.h * a.dist_head_stride);
    const int Dlim = min(g.Dd, a.D);
    float lo[4], hi[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      load_depth_pair(dist_bh, a.dist_pix_stride, g.dpix[k], g.z0, Dlim, g.ok3, lo[k], hi[k]);
    const float hd = 1.f - g.ld;
#pragma unroll
    for (int k = 0; k < 4; ++k) ds[k] = g.ok3 ? lo[k] * hd + hi[k] * g.ld : 0.f;
  } else {
    // no depth-score tensor = plain 2-D multi-scale deformable attention: every in-image corner counts 1
    const float4 t = a.ds_in ? __ldg(reinterpret_cast<const float4 *>(a.ds_in) + (c.pt0 + j))
                             : make_float4(1.f, 1.f, 1.f, 1.f);
    ds[0] = g.pix[0] >= 0 ? t.x : 0.f;
    ds[1] = g.pix[1] >= 0 ? t.y : 0.f;
    ds[2] = g.pix[2] >= 0 ? t.z : 0.f;
    ds[3] = g.pix[3] >= 0 ? t.w : 0.f;
  }
  const int row = a.H * a.C;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float w = aw * (bw[k] * ds[k]);
    if (g.pix[k] >= 0 && w != 0.f) {     // rows that would add nothing are not fetched
      off[k] = g.pix[k] * row;
      wgt[k] = w;
    }
  }
}

// Sums the V channels of a lane over NG groups of G lanes that lie beside each other, and stores them; `out` is where the
// lane's first channel belongs.
template <int V, int G, int NG>
__device__ __forceinline__ void fold_and_store(float (&acc)[V], int lane, float *out, bool live) {
  // 16-bit rows (8 channels a lane): a lane that still holds several values hands half of them over at each exchange, 7
  // shuffles for 32 channels where all of them passed around took 24 (they go through the L1 pipe, which binds), and all
  // lanes write the row (of 16 channels half of them: the fourth exchange has one value left).  The sums are formed in the
  // same order.  bf16, 6 cameras of the base levels: 555 -> 521 us.  For fp32 rows, 3 shuffles instead of 8, it was no gain:
  // 525 -> 529, from offsets 470 -> 481.
  constexpr bool kHalve = V == 8;
  int n = V;
#pragma unroll
  for (int s = G; s < G * NG; s <<= 1) {
    if (kHalve && n > 1) {
      const bool up = lane & s;
      n /= 2;
#pragma unroll
      for (int i = 0; i < n; ++i) {
        const float give = up ? acc[i] : acc[i + n], keep = up ? acc[i + n] : acc[i];
        acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, s);
      }
      if (up) out += n;
    } else {
#pragma unroll
      for (int i = 0; i < n; ++i) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], s);
      live = live && !(lane & s);
    }
  }
  if (!live) return;
  if (n >= 4) {
#pragma unroll
    for (int i = 0; i < n; i += 4)
      *reinterpret_cast<float4 *>(out + i) = make_float4(acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
  } else if (n == 2) {
    *reinterpret_cast<float2 *>(out) = make_float2(acc[0], acc[1]);
  } else {
    *out = acc[0];
  }
}

}  // namespace dfa3d
