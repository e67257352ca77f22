// Row-wise helpers of the encoder layer that surrounds the attention operator (sm_100a):
//
//   * residual add + LayerNorm, forward and backward.  The layer applies `norm(x + branch(x))` after
//     each of its blocks (BEVFormer_DFA3D/projects/mmdet3d_plugin/bevformer/modules/encoder.py:363-411:
//     operation order self_attn, norm, cross_attn, norm, ffn, norm); one kernel reads both summands,
//     writes the sum (the backward needs it) and the normalised rows.
//   * column sums of a (rows, cols) matrix: the bias gradient of a Linear layer.
//
// All three are bound by HBM: every operand is read once and every result written once.  A warp owns a
// row (LayerNorm) or a CTA a band of rows (column sums); per-column results that are summed over rows
// (grad_gamma, grad_beta, the column sums) are accumulated in registers over a CTA's rows, combined in
// shared memory and added to the caller-zeroed output with one `red.global.add.f32` per column and CTA.
#include <stdint.h>

#include <algorithm>

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "dfa3d_launch.h"

namespace dfa3d {
namespace {

constexpr int kLnWarps = 8;
constexpr int kLnThreads = kLnWarps * 32;
constexpr int kCtasPerSm = 4;
constexpr int kSms = 148;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ float4 ld4(const float *p) { return __ldg(reinterpret_cast<const float4 *>(p)); }
// Streaming variants for data touched once.
__device__ __forceinline__ float4 ld4_stream(const float *p) { return __ldcs(reinterpret_cast<const float4 *>(p)); }
__device__ __forceinline__ void st4(float *p, float4 v) { *reinterpret_cast<float4 *>(p) = v; }

// One 16-byte vector reduction into global memory (sm_90+).
__device__ __forceinline__ void red_add_v4(float *addr, float4 v) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(v.x), "f"(v.y), "f"(v.z),
               "f"(v.w)
               : "memory");
}

// Rows of E columns, E a multiple of 4 with 128 * (K - 1) < E <= 128 * K; lane l holds the float4 groups
// l, l + 32, ... of its row (groups at or beyond E are idle).
template <int K>
__global__ void __launch_bounds__(kLnThreads, K <= 4 ? kCtasPerSm : 2)
add_layer_norm_forward_kernel(const float *__restrict__ x, const float *__restrict__ residual,
                              const float *__restrict__ gamma, const float *__restrict__ beta,
                              long long rows, int E, float eps, float *__restrict__ sum_out,
                              float *__restrict__ y, float *__restrict__ mean_out,
                              float *__restrict__ rstd_out) {
  const float inv_e = 1.f / (float)E;
  const int lane = threadIdx.x & 31;
  const long long warp0 = (long long)blockIdx.x * kLnWarps + (threadIdx.x >> 5);
  const long long stride = (long long)gridDim.x * kLnWarps;
  for (long long row = warp0; row < rows; row += stride) {
    const float *xr = x + row * E;
    float4 v[K];
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const int c = (lane + 32 * j) * 4;
      v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c >= E) continue;
      v[j] = ld4_stream(xr + c);
      if (residual) {
        const float4 r = ld4_stream(residual + row * E + c);
        v[j].x += r.x; v[j].y += r.y; v[j].z += r.z; v[j].w += r.w;
      }
      s += (v[j].x + v[j].y) + (v[j].z + v[j].w);
    }
    const float mean = warp_sum(s) * inv_e;
    float q = 0.f;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      if ((lane + 32 * j) * 4 >= E) continue;
      const float a = v[j].x - mean, b = v[j].y - mean, c = v[j].z - mean, d = v[j].w - mean;
      q += (a * a + b * b) + (c * c + d * d);
    }
    const float rstd = rsqrtf(warp_sum(q) * inv_e + eps);
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const int c = (lane + 32 * j) * 4;
      if (c >= E) continue;
      if (sum_out) st4(sum_out + row * E + c, v[j]);
      const float4 g = ld4(gamma + c), b = ld4(beta + c);
      float4 o;
      o.x = (v[j].x - mean) * rstd * g.x + b.x;
      o.y = (v[j].y - mean) * rstd * g.y + b.y;
      o.z = (v[j].z - mean) * rstd * g.z + b.z;
      o.w = (v[j].w - mean) * rstd * g.w + b.w;
      st4(y + row * E + c, o);
    }
    if (lane == 0 && mean_out) {        // no backward will ask for them otherwise
      mean_out[row] = mean;
      rstd_out[row] = rstd;
    }
  }
}

// grad_in = rstd * (g*gamma - mean(g*gamma) - xhat * mean(g*gamma*xhat)); grad_gamma += g*xhat;
// grad_beta += g, both summed over rows.
template <int K>
__global__ void __launch_bounds__(kLnThreads, K <= 1 ? kCtasPerSm : (K == 2 ? 3 : (K <= 4 ? 2 : 1)))
layer_norm_backward_kernel(const float *__restrict__ grad_y, const float *__restrict__ in,
                           const float *__restrict__ gamma, const float *__restrict__ mean_in,
                           const float *__restrict__ rstd_in, long long rows, int E,
                           float *__restrict__ grad_in, float *__restrict__ grad_gamma,
                           float *__restrict__ grad_beta) {
  const float inv_e = 1.f / (float)E;
  __shared__ float4 part[kLnWarps][32 * K];      // one warp's per-column partial sums
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long warp0 = (long long)blockIdx.x * kLnWarps + warp;
  const long long stride = (long long)gridDim.x * kLnWarps;
  float4 dg[K], db[K];
#pragma unroll
  for (int j = 0; j < K; ++j) {
    dg[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    db[j] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  // R rows of a warp are in flight together (narrow rows leave registers for it): their loads are issued
  // before any of them is reduced
  constexpr int R = K <= 2 ? 2 : 1;
  for (long long row0 = warp0; row0 < rows; row0 += stride * R) {
    float4 g[R][K], xh[R][K];
    float mean[R], rstd[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const long long row = row0 + r * stride;
      const bool live = row < rows;
      mean[r] = live ? __ldg(mean_in + row) : 0.f;
      rstd[r] = live ? __ldg(rstd_in + row) : 0.f;
#pragma unroll
      for (int j = 0; j < K; ++j) {
        const int c = (lane + 32 * j) * 4;
        g[r][j] = make_float4(0.f, 0.f, 0.f, 0.f);
        xh[r][j] = g[r][j];
        if (live && c < E) {
          g[r][j] = ld4_stream(grad_y + row * E + c);
          xh[r][j] = ld4_stream(in + row * E + c);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const long long row = row0 + r * stride;
      if (row >= rows) break;
      float s1 = 0.f, s2 = 0.f;
#pragma unroll
      for (int j = 0; j < K; ++j) {
        const int c = (lane + 32 * j) * 4;
        if (c >= E) continue;
        float4 &G = g[r][j], &X = xh[r][j];
        X = make_float4((X.x - mean[r]) * rstd[r], (X.y - mean[r]) * rstd[r], (X.z - mean[r]) * rstd[r],
                        (X.w - mean[r]) * rstd[r]);
        dg[j].x += G.x * X.x; dg[j].y += G.y * X.y; dg[j].z += G.z * X.z; dg[j].w += G.w * X.w;
        db[j].x += G.x; db[j].y += G.y; db[j].z += G.z; db[j].w += G.w;
        const float4 gam = ld4(gamma + c);
        G.x *= gam.x; G.y *= gam.y; G.z *= gam.z; G.w *= gam.w;
        s1 += (G.x + G.y) + (G.z + G.w);
        s2 += (G.x * X.x + G.y * X.y) + (G.z * X.z + G.w * X.w);
      }
      const float c1 = warp_sum(s1) * inv_e, c2 = warp_sum(s2) * inv_e;
#pragma unroll
      for (int j = 0; j < K; ++j) {
        const int c = (lane + 32 * j) * 4;
        if (c >= E) continue;
        const float4 G = g[r][j], X = xh[r][j];
        float4 o;
        o.x = rstd[r] * (G.x - c1 - X.x * c2);
        o.y = rstd[r] * (G.y - c1 - X.y * c2);
        o.z = rstd[r] * (G.z - c1 - X.z * c2);
        o.w = rstd[r] * (G.w - c1 - X.w * c2);
        st4(grad_in + row * E + c, o);
      }
    }
  }
  // combine the CTA's warps, then one reduction per column and CTA; gamma first, beta second
#pragma unroll
  for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
    for (int j = 0; j < K; ++j) part[warp][lane + 32 * j] = pass == 0 ? dg[j] : db[j];
    __syncthreads();
    float *dst = pass == 0 ? grad_gamma : grad_beta;
    for (int c4 = threadIdx.x; c4 * 4 < E; c4 += kLnThreads) {
      float4 t = part[0][c4];
#pragma unroll
      for (int w = 1; w < kLnWarps; ++w) {
        const float4 u = part[w][c4];
        t.x += u.x; t.y += u.y; t.z += u.z; t.w += u.w;
      }
      red_add_v4(dst + c4 * 4, t);
    }
    __syncthreads();
  }
}

// Column sums: a CTA is 64 float4 column groups x 8 row lanes; blockIdx.y picks the band of 256 columns,
// blockIdx.x the rows (grid-strided).  dst is accumulated into (caller-zeroed).  Few, long-lived CTAs: every
// CTA ends with one vector reduction per column group into the same few sectors of dst, and those
// serialise in L2.
constexpr int kCsGroups = 64, kCsLanes = 8, kCsThreads = kCsGroups * kCsLanes;

__global__ void __launch_bounds__(kCsThreads)
column_sum_kernel(const float *__restrict__ src, long long rows, int cols, float *__restrict__ dst) {
  __shared__ float4 part[kCsLanes][kCsGroups];
  const int grp = threadIdx.x % kCsGroups, rl = threadIdx.x / kCsGroups;
  const int col = (blockIdx.y * kCsGroups + grp) * 4;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  if (col < cols) {
    const long long step = (long long)gridDim.x * kCsLanes;
    long long r = (long long)blockIdx.x * kCsLanes + rl;
    // four independent loads in flight per thread
    for (; r + 3 * step < rows; r += 4 * step) {
      const float4 a = ld4_stream(src + r * cols + col), b = ld4_stream(src + (r + step) * cols + col);
      const float4 c = ld4_stream(src + (r + 2 * step) * cols + col);
      const float4 d = ld4_stream(src + (r + 3 * step) * cols + col);
      acc.x += (a.x + b.x) + (c.x + d.x); acc.y += (a.y + b.y) + (c.y + d.y);
      acc.z += (a.z + b.z) + (c.z + d.z); acc.w += (a.w + b.w) + (c.w + d.w);
    }
    for (; r < rows; r += step) {
      const float4 a = ld4_stream(src + r * cols + col);
      acc.x += a.x; acc.y += a.y; acc.z += a.z; acc.w += a.w;
    }
  }
  part[rl][grp] = acc;
  __syncthreads();
  if (rl == 0 && col < cols) {
    float4 t = part[0][grp];
#pragma unroll
    for (int i = 1; i < kCsLanes; ++i) {
      t.x += part[i][grp].x; t.y += part[i][grp].y; t.z += part[i][grp].z; t.w += part[i][grp].w;
    }
    red_add_v4(dst + col, t);
  }
}

// Backward of relu(x W^T + b) up to the products: grad_in = y <= 0 ? 0 : grad_y (a NaN lets its gradient pass, as in
// torch) and its column sums (the bias gradient) in one pass over both operands.  Split and accumulation as in column_sum_kernel.
__global__ void __launch_bounds__(kCsThreads)
relu_backward_kernel(const float *grad_y, const float *__restrict__ y, long long rows, int cols,
                     float *grad_in, float *__restrict__ dst) {
  __shared__ float4 part[kCsLanes][kCsGroups];
  const int grp = threadIdx.x % kCsGroups, rl = threadIdx.x / kCsGroups;
  const int col = (blockIdx.y * kCsGroups + grp) * 4;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  if (col < cols) {
    const long long step = (long long)gridDim.x * kCsLanes;
    constexpr int U = 4;
    for (long long r = (long long)blockIdx.x * kCsLanes + rl; r < rows; r += U * step) {
      float4 g[U], v[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (r + u * step < rows) {
          g[u] = ld4_stream(grad_y + (r + u * step) * cols + col);
          v[u] = ld4_stream(y + (r + u * step) * cols + col);
        }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (r + u * step < rows) {
          const float4 t = make_float4(v[u].x <= 0.f ? 0.f : g[u].x, v[u].y <= 0.f ? 0.f : g[u].y,
                                       v[u].z <= 0.f ? 0.f : g[u].z, v[u].w <= 0.f ? 0.f : g[u].w);
          st4(grad_in + (r + u * step) * cols + col, t);
          acc.x += t.x; acc.y += t.y; acc.z += t.z; acc.w += t.w;
        }
    }
  }
  part[rl][grp] = acc;
  __syncthreads();
  if (rl == 0 && col < cols) {
    float4 t = part[0][grp];
#pragma unroll
    for (int i = 1; i < kCsLanes; ++i) {
      t.x += part[i][grp].x; t.y += part[i][grp].y; t.z += part[i][grp].z; t.w += part[i][grp].w;
    }
    red_add_v4(dst + col, t);
  }
}

// Last step of a weight gradient formed as a batch of row slices: dst (out, in) = sum of the `slices` partial products,
// plus the outer products of the few rows that no slice covers.  Zeroes the bias gradient on the way (the column sum that
// follows accumulates into it): one launch instead of a reduction, a product of 15 rows and a fill.  Bound by reading the
// slices.
__global__ void __launch_bounds__(256)
slice_sum_kernel(const float *__restrict__ part, int slices, int out, int in, const float *__restrict__ g_tail,
                 const float *__restrict__ x_tail, int tail, float *__restrict__ dst, float *__restrict__ zero) {
  const long long n4 = (long long)out * in / 4, t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (zero && t < out) zero[t] = 0.f;
  if (t >= n4) return;
  float4 acc = ld4_stream(part + t * 4);
  int s = 1;
  constexpr int U = 5;                       // 16 slices: three rounds of five
  for (; s + U <= slices; s += U) {
    float4 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = ld4_stream(part + ((s + u) * n4 + t) * 4);
#pragma unroll
    for (int u = 0; u < U; ++u) { acc.x += v[u].x; acc.y += v[u].y; acc.z += v[u].z; acc.w += v[u].w; }
  }
  for (; s < slices; ++s) {
    const float4 v = ld4_stream(part + (s * n4 + t) * 4);
    acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
  }
  const int o = (int)(t * 4 / in), i = (int)(t * 4 - (long long)o * in);
#pragma unroll 5
  for (int r = 0; r < tail; ++r) {
    const float g = __ldg(g_tail + (long long)r * out + o);
    const float4 x = ld4(x_tail + (long long)r * in + i);
    acc.x = fmaf(g, x.x, acc.x); acc.y = fmaf(g, x.y, acc.y); acc.z = fmaf(g, x.z, acc.z); acc.w = fmaf(g, x.w, acc.w);
  }
  st4(dst + t * 4, acc);
}

// Up to eight buffers, one after the other, into as many places: the weights and biases of Linear layers that are run as
// one.
struct Segments {
  const float *src[8];
  float *dst[8];
  long long n[8];
};
__global__ void __launch_bounds__(256) copy_segments_kernel(const Segments s) {
  const float *src = s.src[blockIdx.y];
  float *dst = s.dst[blockIdx.y];
  const long long n = s.n[blockIdx.y], step = (long long)gridDim.x * blockDim.x;
  const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const bool vec = ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15u) == 0;
  const long long n4 = vec ? n >> 2 : 0;
  for (long long t = t0; t < n4; t += step) st4(dst + t * 4, ld4(src + t * 4));
  for (long long t = n4 * 4 + t0; t < n; t += step) dst[t] = __ldg(src + t);
}

// Zeroes two buffers with one launch (a backward zeroes the two gradients it accumulates into; for a small
// problem a second fill is a launch gap longer than the fill).  16-byte stores, the ragged ends one by one.
__global__ void __launch_bounds__(256) zero_two_kernel(float *a, long long na, float *b, long long nb) {
  const long long va = na >> 2, vb = nb >> 2, step = (long long)gridDim.x * blockDim.x;
  const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  for (long long t = t0; t < va + vb; t += step)
    st4(t < va ? a + t * 4 : b + (t - va) * 4, make_float4(0.f, 0.f, 0.f, 0.f));
  if (t0 < (na & 3)) a[va * 4 + t0] = 0.f;
  if (t0 < (nb & 3)) b[vb * 4 + t0] = 0.f;
}

// Converts up to two buffers between fp32 and a 16-bit type with one launch, eight elements (16 bytes of the narrow type) a
// thread at a time, the ragged ends one by one.  Bound by HBM and L2.  The five conversions of an fp16 operator call and its
// backward (outputs 6.9 M elements, gradients 4.2 M, grad_out 1.5 M), one launch of torch's each: 20.7 us; as three 14.4.
template <typename T> struct Narrow;
template <> struct Narrow<__half> {
  __device__ static __forceinline__ __half of(float x) { return __float2half_rn(x); }
  __device__ static __forceinline__ float wide(__half x) { return __half2float(x); }
};
template <> struct Narrow<__nv_bfloat16> {
  __device__ static __forceinline__ __nv_bfloat16 of(float x) { return __float2bfloat16_rn(x); }
  __device__ static __forceinline__ float wide(__nv_bfloat16 x) { return __bfloat162float(x); }
};

template <typename T, bool WIDEN>
__global__ void __launch_bounds__(256)
convert_two_kernel(void *n0, void *w0, long long c0, void *n1, void *w1, long long c1) {
  const long long v0 = c0 >> 3, v1 = c1 >> 3, step = (long long)gridDim.x * blockDim.x;
  const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  for (long long t = t0; t < v0 + v1; t += step) {
    T *n = t < v0 ? static_cast<T *>(n0) + t * 8 : static_cast<T *>(n1) + (t - v0) * 8;
    float *w = t < v0 ? static_cast<float *>(w0) + t * 8 : static_cast<float *>(w1) + (t - v0) * 8;
    __align__(16) T x[8];
    if (WIDEN) {
      *reinterpret_cast<uint4 *>(x) = *reinterpret_cast<const uint4 *>(n);
#pragma unroll
      for (int i = 0; i < 8; i += 4)
        st4(w + i, make_float4(Narrow<T>::wide(x[i]), Narrow<T>::wide(x[i + 1]), Narrow<T>::wide(x[i + 2]),
                               Narrow<T>::wide(x[i + 3])));
    } else {
#pragma unroll
      for (int i = 0; i < 8; i += 4) {
        const float4 f = *reinterpret_cast<const float4 *>(w + i);
        x[i] = Narrow<T>::of(f.x); x[i + 1] = Narrow<T>::of(f.y); x[i + 2] = Narrow<T>::of(f.z); x[i + 3] = Narrow<T>::of(f.w);
      }
      *reinterpret_cast<uint4 *>(n) = *reinterpret_cast<const uint4 *>(x);
    }
  }
  auto one = [&](void *n, void *w, long long i) {
    if (WIDEN) static_cast<float *>(w)[i] = Narrow<T>::wide(static_cast<const T *>(n)[i]);
    else static_cast<T *>(n)[i] = Narrow<T>::of(static_cast<const float *>(w)[i]);
  };
  if (t0 < (c0 & 7)) one(n0, w0, v0 * 8 + t0);
  if (t0 < (c1 & 7)) one(n1, w1, v1 * 8 + t0);
}

unsigned row_grid(long long rows) {
  const long long want = (rows + kLnWarps - 1) / kLnWarps;
  const long long cap = (long long)kSms * kCtasPerSm;
  return (unsigned)(want < cap ? (want > 0 ? want : 1) : cap);
}

}  // namespace

int layer_norm_max_columns() { return 1024; }

cudaError_t launch_add_layer_norm_forward(const float *x, const float *residual, const float *gamma,
                                          const float *beta, long long rows, int E, float eps,
                                          float *sum_out, float *y, float *mean, float *rstd,
                                          cudaStream_t s) {
  if (rows == 0) return cudaSuccess;
  const unsigned grid = row_grid(rows);
#define DFA3D_LN_FWD(K)                                                                              \
  case K:                                                                                            \
    add_layer_norm_forward_kernel<K><<<grid, kLnThreads, 0, s>>>(x, residual, gamma, beta, rows, E,  \
                                                                 eps, sum_out, y, mean, rstd);       \
    break;
  switch ((E + 127) / 128) {
    DFA3D_LN_FWD(1) DFA3D_LN_FWD(2) DFA3D_LN_FWD(3) DFA3D_LN_FWD(4)
    DFA3D_LN_FWD(5) DFA3D_LN_FWD(6) DFA3D_LN_FWD(7) DFA3D_LN_FWD(8)
    default: return cudaErrorInvalidValue;
  }
#undef DFA3D_LN_FWD
  return cudaGetLastError();
}

cudaError_t launch_layer_norm_backward(const float *grad_y, const float *in, const float *gamma,
                                       const float *mean, const float *rstd, long long rows, int E,
                                       float *grad_in, float *grad_gamma, float *grad_beta,
                                       cudaStream_t s) {
  if (rows == 0) return cudaSuccess;
  // as many CTAs as are resident at once (the kernel's launch bounds), each with at least 8 rows per warp:
  // every CTA ends with E/4 vector reductions per output
  const int K = (E + 127) / 128;
  const long long want = (rows + kLnWarps * 8 - 1) / (kLnWarps * 8);
  const long long cap = (long long)kSms * (K <= 1 ? kCtasPerSm : (K == 2 ? 3 : (K <= 4 ? 2 : 1)));
  const unsigned grid = (unsigned)(want < cap ? (want > 0 ? want : 1) : cap);
#define DFA3D_LN_BWD(K)                                                                               \
  case K:                                                                                             \
    layer_norm_backward_kernel<K><<<grid, kLnThreads, 0, s>>>(grad_y, in, gamma, mean, rstd, rows, E,  \
                                                              grad_in, grad_gamma, grad_beta);        \
    break;
  switch (K) {
    DFA3D_LN_BWD(1) DFA3D_LN_BWD(2) DFA3D_LN_BWD(3) DFA3D_LN_BWD(4)
    DFA3D_LN_BWD(5) DFA3D_LN_BWD(6) DFA3D_LN_BWD(7) DFA3D_LN_BWD(8)
    default: return cudaErrorInvalidValue;
  }
#undef DFA3D_LN_BWD
  return cudaGetLastError();
}

cudaError_t launch_column_sum(const float *src, long long rows, int cols, float *dst, cudaStream_t s) {
  if (rows == 0 || cols == 0) return cudaSuccess;
  const unsigned bands = (unsigned)((cols / 4 + kCsGroups - 1) / kCsGroups);
  long long gx = (long long)kSms * 2 / bands;                            // two 512-thread CTAs per SM
  const long long most = (rows + kCsLanes * 8 - 1) / (kCsLanes * 8);     // at least 8 rows per thread
  if (gx > most) gx = most;
  if (gx < 1) gx = 1;
  column_sum_kernel<<<dim3((unsigned)gx, bands, 1), kCsThreads, 0, s>>>(src, rows, cols, dst);
  return cudaGetLastError();
}

cudaError_t launch_relu_backward(const float *grad_y, const float *y, long long rows, int cols, float *grad_in, float *dst,
                                 cudaStream_t s) {
  if (rows == 0 || cols == 0) return cudaSuccess;
  const unsigned bands = (unsigned)((cols / 4 + kCsGroups - 1) / kCsGroups);
  long long gx = (long long)kSms * 2 / bands;                            // as launch_column_sum
  const long long most = (rows + kCsLanes * 8 - 1) / (kCsLanes * 8);
  if (gx > most) gx = most;
  if (gx < 1) gx = 1;
  relu_backward_kernel<<<dim3((unsigned)gx, bands, 1), kCsThreads, 0, s>>>(grad_y, y, rows, cols, grad_in, dst);
  return cudaGetLastError();
}

cudaError_t launch_slice_sum(const float *part, int slices, int out, int in, const float *g_tail, const float *x_tail, int tail,
                             float *dst, float *zero, cudaStream_t s) {
  const long long n = std::max((long long)out * in / 4, (long long)out);
  slice_sum_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(part, slices, out, in, g_tail, x_tail, tail, dst, zero);
  return cudaGetLastError();
}

cudaError_t launch_copy_segments(const float *const *src, float *const *dst, const long long *n, int count, cudaStream_t s) {
  Segments g;
  long long most = 0;
  for (int i = 0; i < count; ++i) {
    g.src[i] = src[i]; g.dst[i] = dst[i]; g.n[i] = n[i];
    most = std::max(most, n[i]);
  }
  if (most == 0) return cudaSuccess;
  const unsigned gx = (unsigned)std::min((most / 4 + 255) / 256 + 1, 148LL * 2);
  copy_segments_kernel<<<dim3(gx, (unsigned)count), 256, 0, s>>>(g);
  return cudaGetLastError();
}

cudaError_t launch_zero_two(float *a, long long na, float *b, long long nb, cudaStream_t s) {
  const long long groups = (na + nb + 3) / 4, want = (groups + 255) / 256, cap = (long long)kSms * 8;
  if (na + nb == 0) return cudaSuccess;
  zero_two_kernel<<<(unsigned)(want < cap ? want : cap), 256, 0, s>>>(a, na, b, nb);
  return cudaGetLastError();
}

cudaError_t launch_convert_two(bool half, bool widen, void *n0, void *w0, long long c0, void *n1, void *w1, long long c1,
                               cudaStream_t s) {
  if (c0 + c1 == 0) return cudaSuccess;
  const long long want = ((c0 + c1 + 7) / 8 + 255) / 256, cap = (long long)kSms * 8;
  const unsigned grid = (unsigned)(want < cap ? want : cap);
  if (half && widen) convert_two_kernel<__half, true><<<grid, 256, 0, s>>>(n0, w0, c0, n1, w1, c1);
  else if (half) convert_two_kernel<__half, false><<<grid, 256, 0, s>>>(n0, w0, c0, n1, w1, c1);
  else if (widen) convert_two_kernel<__nv_bfloat16, true><<<grid, 256, 0, s>>>(n0, w0, c0, n1, w1, c1);
  else convert_two_kernel<__nv_bfloat16, false><<<grid, 256, 0, s>>>(n0, w0, c0, n1, w1, c1);
  return cudaGetLastError();
}

}  // namespace dfa3d
