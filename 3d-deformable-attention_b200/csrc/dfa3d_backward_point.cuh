// Backward of one sampling point and the reduction of its rows' dot products: shared by the kernels with one item per
// warp and with several.
#pragma once
#include "dfa3d_common.cuh"

namespace dfa3d {

// Per-lane state of one sampling point that the epilogue needs.
struct PointState {
  PointGeo g;
  float aw;
  float bw[4], ds[4];
  float dz[4];          // dist[z0+1] - dist[z0] per corner (fused mode): d depth_score / d depth
  bool live;            // j < LP && ok2
};

template <typename DT, int MODE>
__device__ __forceinline__ void bwd_point(const KArgs &a, const LevelTable &lv, const ItemCtx &c, int j,
                                          const SoftmaxStats &sm, PointState &s, float (&wgt)[4],
                                          int (&off)[4]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    s.ds[k] = 0.f; s.bw[k] = 0.f; s.dz[k] = 0.f; wgt[k] = 0.f; off[k] = -1;
    s.g.pix[k] = -1; s.g.dpix[k] = -1;
  }
  s.live = false; s.aw = 0.f; s.g.ok2 = false; s.g.ok3 = false;
  if (j >= a.LP) return;
  const int l = j / a.P;
  float x, y, z;
  read_point<MODE>(a, lv, c, j, l, sm, x, y, z, s.aw);
  s.g = point_geometry(x, y, z, mode_has_depth(MODE), lv.h[l], lv.w[l], lv.d[l], lv.start[l], a.N,
                       dist_map_of(a, lv, l));
  if (!s.g.ok2) return;
  s.live = true;
  bilinear_weights(s.g, s.bw);
  if (mode_has_depth(MODE)) {
    const DT *dist_bh = reinterpret_cast<const DT *>(a.dist) +
                        ((long long)c.b * a.Nd * a.dist_pix_stride + c.h * a.dist_head_stride);
    const int Dlim = min(s.g.Dd, a.D);
    float lo[4], hi[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      load_depth_pair(dist_bh, a.dist_pix_stride, s.g.dpix[k], s.g.z0, Dlim, s.g.ok3, lo[k], hi[k]);
    const float hd = 1.f - s.g.ld;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      s.ds[k] = s.g.ok3 ? lo[k] * hd + hi[k] * s.g.ld : 0.f;
      s.dz[k] = hi[k] - lo[k];
    }
  } else {
    const float4 t = a.ds_in ? __ldg(reinterpret_cast<const float4 *>(a.ds_in) + (c.pt0 + j))
                             : make_float4(1.f, 1.f, 1.f, 1.f);
    s.ds[0] = s.g.pix[0] >= 0 ? t.x : 0.f;
    s.ds[1] = s.g.pix[1] >= 0 ? t.y : 0.f;
    s.ds[2] = s.g.pix[2] >= 0 ? t.z : 0.f;
    s.ds[3] = s.g.pix[3] >= 0 ? t.w : 0.f;
  }
  const int row = a.H * a.C;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (s.g.pix[k] >= 0) {
      off[k] = s.g.pix[k] * row;
      wgt[k] = s.aw * (s.bw[k] * s.ds[k]);
    }
}

// Everything that follows from the four dot products t[k] = <value row k, grad_out row>.
// Returns attention weight x its gradient (the point's term of the softmax-backward dot product;
// used in caller-fused mode only).
template <typename DT, int MODE>
__device__ __forceinline__ float bwd_point_epilogue(const KArgs &a, const ItemCtx &c, int j,
                                                    const PointState &s, const float (&t)[4]) {
  if (j >= a.LP) return 0.f;
  const long long pt = c.pt0 + j;
  float g_attn = 0.f, g_x = 0.f, g_y = 0.f, g_z = 0.f;
  float gds[4] = {0.f, 0.f, 0.f, 0.f};
  if (s.live) {
    const float hw = 1.f - s.g.lw, hh = 1.f - s.g.lh;
    float tt[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) tt[k] = s.g.pix[k] >= 0 ? t[k] : 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      g_attn = fmaf(s.bw[k] * s.ds[k], tt[k], g_attn);
      gds[k] = s.g.pix[k] >= 0 ? s.aw * (s.bw[k] * tt[k]) : 0.f;
    }
    const float e0 = s.ds[0] * tt[0], e1 = s.ds[1] * tt[1], e2 = s.ds[2] * tt[2], e3 = s.ds[3] * tt[3];
    g_x = (float)s.g.W * s.aw * (hh * (e1 - e0) + s.g.lh * (e2 - e3));
    g_y = (float)s.g.Hh * s.aw * (hw * (e3 - e0) + s.g.lw * (e2 - e1));
    if (mode_has_depth(MODE) && s.g.ok3) {
      float *gd_bh = a.grad_dist + ((long long)c.b * a.Nd * a.dist_pix_stride + c.h * a.dist_head_stride);
      const float hd = 1.f - s.g.ld;
      const int Dlim = min(s.g.Dd, a.D);
      float acc = 0.f;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (s.g.pix[k] >= 0) {
          if (gds[k] != 0.f)
            red_depth_pair(gd_bh, a.dist_pix_stride, s.g.dpix[k], s.g.z0, Dlim, a.D, hd * gds[k],
                           s.g.ld * gds[k]);
          acc = fmaf(gds[k], s.dz[k], acc);
        }
      }
      g_z = (float)s.g.Dd * acc;
    }
  }
  if (mode_from_offsets(MODE)) {
    // d loc / d offset = 1 / (W, H, D); the logit gradient needs the whole item's dot product and is
    // finished by finish_logit_grads(): park the attention gradient in its slot for now
    const long long lg = (c.attn - a.attn) + j;
    a.grad_attn[lg] = g_attn;
    float *gu = a.grad_loc + (c.loc - a.loc) + j * 2;
    gu[0] = s.live ? __fdiv_rn(g_x, (float)s.g.W) : 0.f;
    gu[1] = s.live ? __fdiv_rn(g_y, (float)s.g.Hh) : 0.f;
    if (MODE == kCallerFused) a.grad_off_d[lg] = __fdiv_rn(g_z, (float)a.D);
    return s.aw * g_attn;
  }
  a.grad_attn[pt] = g_attn;
  float *gl = a.grad_loc + pt * a.loc_stride;
  gl[0] = g_x;
  gl[1] = g_y;
  if (MODE == kFused) gl[2] = g_z;
  if (a.grad_ds_out)
    reinterpret_cast<float4 *>(a.grad_ds_out)[pt] = make_float4(gds[0], gds[1], gds[2], gds[3]);
  return 0.f;
}

// Dot products of U = 4 row fragments with the grad_out fragment, summed over the G >= 4 lanes of a group.
// The four sums are folded together: after the first exchange a lane keeps two of them, after the second one, and the
// rest is a butterfly: 3, 4, 5 or 6 shuffles for G = 4, 8, 16, 32 instead of 8, 12, 16 or 20.  Lane `sub` < 4 of every
// group ends up with the total of row u = 2*(sub & 1) + ((sub >> 1) & 1).  Shuffles travel through the same pipe as the
// shared-memory and global accesses these kernels are bound by.
// Returns the lane's total and, in `u_mine`, which of the four rows it belongs to (-1: none).
template <int G>
__device__ __forceinline__ float fold_four_dots(const float (&d)[4], int sub, int &u_mine) {
  const bool b0 = sub & 1, b1 = sub & 2;
  const float r0 = __shfl_xor_sync(0xffffffffu, b0 ? d[0] : d[2], 1);
  const float r1 = __shfl_xor_sync(0xffffffffu, b0 ? d[1] : d[3], 1);
  const float e0 = (b0 ? d[2] : d[0]) + r0, e1 = (b0 ? d[3] : d[1]) + r1;
  const float r2 = __shfl_xor_sync(0xffffffffu, b1 ? e0 : e1, 2);
  float f = (b1 ? e1 : e0) + r2;
#pragma unroll
  for (int s = 4; s < G; s <<= 1) f += __shfl_xor_sync(0xffffffffu, f, s);
  u_mine = sub < 4 ? (b0 ? 2 : 0) + (b1 ? 1 : 0) : -1;
  return f;
}

}  // namespace dfa3d
