// Producer of the depth distribution in the operator's layout (sm_100a).
//
// The depth network ends in a (B, D, hs, ws) map of logits.  The reference turns it into what the
// attention reads in four steps, each a pass over HBM: softmax (or sigmoid) over the D channels
// (BEVFormer_DFA3D/projects/mmdet3d_plugin/bevformer/dense_heads/depth_head.py:265-268), one
// F.interpolate(mode="nearest") per feature level (:273-276), flatten + permute + cat of the levels
// (…/modules/transformer.py:368-391) and the permute to (bs*cams, sum hw, D) of the spatial
// cross-attention (spatial_cross_attention.py:727-728).  Here one kernel reads the logits once and
// writes dist (B, N, D) -- fp32, bf16 or fp16 -- for all levels, channel-last; its backward reads the
// gradient of that tensor and the logits once and writes the gradient of the logits.
//
// Nearest resize, as torch computes it: source index = min(floor(dst * scale), size - 1) with
// scale = (float)source size / (float)level size.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include "dfa3d_b200.h"
#include "dfa3d_launch.h"

namespace dfa3d {
namespace {

constexpr int kTile = 32;          // map pixels of one map row per CTA
constexpr int kMaxBins = 256;      // D limit of the shared-memory tile
constexpr int kProdThreads = 256;
constexpr int kProdLevels = DFA3D_MAX_LEVELS;

struct ProdArgs {
  const float *logits;      // (B, D, hs, ws)
  const int64_t *shapes;    // (L, shape_stride) int64: (h, w, ...) per level
  const int64_t *lsi;       // (L) int64
  void *dist;               // (B, N, D) fp32 | bf16 | fp16
  const void *grad_dist;    // (B, N, D) fp32 | bf16 | fp16
  float *grad_logits;       // (B, D, hs, ws)
  int B, D, hs, ws, N, L, shape_stride;
  int sigmoid;              // 0: softmax over D, 1: element-wise sigmoid
};

__device__ __forceinline__ int nearest_src(int dst, float scale, int size) {
  return min((int)floorf((float)dst * scale), size - 1);
}

// V neighbouring bins of a dist row with one access; widened to / narrowed from fp32.  V = 4 or 2 needs a D that is a
// multiple of it (rows then start on V bins).
template <typename T, int V> struct Word;
template <> struct Word<float, 4> { using type = float4; };
template <> struct Word<float, 2> { using type = float2; };
template <> struct Word<float, 1> { using type = float; };
template <> struct Word<__nv_bfloat16, 4> { using type = uint2; };
template <> struct Word<__nv_bfloat16, 2> { using type = uint32_t; };
template <> struct Word<__nv_bfloat16, 1> { using type = unsigned short; };
template <> struct Word<__half, 4> { using type = uint2; };
template <> struct Word<__half, 2> { using type = uint32_t; };
template <> struct Word<__half, 1> { using type = unsigned short; };

__device__ __forceinline__ float narrow(float, float v) { return v; }
__device__ __forceinline__ __nv_bfloat16 narrow(__nv_bfloat16, float v) { return __float2bfloat16_rn(v); }
__device__ __forceinline__ __half narrow(__half, float v) { return __float2half_rn(v); }
__device__ __forceinline__ float widen(float v) { return v; }
__device__ __forceinline__ float widen(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float widen(__half v) { return __half2float(v); }

template <int V, typename T>
__device__ __forceinline__ void load_bins(const T *p, float (&r)[V]) {
  union { typename Word<T, V>::type w; T t[V]; } u;
  u.w = __ldg(reinterpret_cast<const typename Word<T, V>::type *>(p));
#pragma unroll
  for (int i = 0; i < V; ++i) r[i] = widen(u.t[i]);
}
// the bins as they are stored, formed once for all the rows that receive them
template <typename T, int V>
__device__ __forceinline__ typename Word<T, V>::type pack_bins(const float (&v)[V]) {
  union { typename Word<T, V>::type w; T t[V]; } u;
#pragma unroll
  for (int i = 0; i < V; ++i) u.t[i] = narrow(T(), v[i]);
  return u.w;
}

// Smallest dst in [0, n] whose nearest source is at or past s (n: none is).  The resize is monotone.
__device__ __forceinline__ int first_at(int s, float scale, int n, int size) {
  if (s >= size) return n;
  int d = min(n, max(0, (int)((float)s / scale) - 2));
  while (d > 0 && nearest_src(d - 1, scale, size) >= s) --d;
  while (d < n && nearest_src(d, scale, size) < s) ++d;
  return d;
}

// Which level pixels read the CTA's map pixels (row sy, columns sx0 .. sx0 + kTile - 1): per level the rows
// [y0, y1) and, per map pixel i, the columns [x[i], x[i+1]).
struct Footprint {
  int4 level[kProdLevels];           // y0, y1, width, first row of dist
  int x[kProdLevels][kTile + 1];
};

__device__ __forceinline__ void stage_footprint(Footprint &f, const ProdArgs &a, int sy, int sx0) {
  for (int t = threadIdx.x; t < a.L * (kTile + 2); t += kProdThreads) {
    const int l = t / (kTile + 2), i = t - l * (kTile + 2);
    const int w = (int)a.shapes[l * a.shape_stride + 1];
    if (i <= kTile) {
      f.x[l][i] = first_at(min(sx0 + i, a.ws), (float)a.ws / (float)w, w, a.ws);
    } else {
      const int h = (int)a.shapes[l * a.shape_stride];
      const float scale = (float)a.hs / (float)h;
      f.level[l] = make_int4(first_at(sy, scale, h, a.hs), first_at(sy + 1, scale, h, a.hs), w, (int)a.lsi[l]);
    }
  }
}

// Calls row(n) for every row n of dist that reads map pixel i of the CTA, levels, rows and columns in order.
template <typename F>
__device__ __forceinline__ void for_each_row(const Footprint &f, const ProdArgs &a, int i, F row) {
  for (int l = 0; l < a.L; ++l) {
    const int x0 = f.x[l][i], nx = f.x[l][i + 1] - x0;
    const int4 v = f.level[l];
    if (nx == 0) continue;
    for (int y = v.x; y < v.y; ++y) {
      const int n = v.w + y * v.z + x0;
      for (int x = 0; x < nx; ++x)
        if ((unsigned)(n + x) < (unsigned)a.N) row(n + x);
    }
  }
}

// The tile: row i holds the bins of map pixel i, padded to a multiple of four; rows start four words apart modulo 32
// banks, so that 16-byte accesses are free of conflicts both along a row and from row to row.
__host__ __device__ __forceinline__ int padded(int D) { return (D + 3) & ~3; }
__host__ __device__ __forceinline__ int tile_stride(int D) { return (padded(D) + 31) / 32 * 32 + 4; }

// Logits of the CTA's map pixels into the tile (padding: -inf, so that it vanishes in the softmax).  A thread takes
// four bins of one pixel: four loads along the map's x axis, one 16-byte store.
__device__ __forceinline__ void load_tile(float *tile, int stride, const ProdArgs &a, const float *lg, int npix) {
  const long long plane = (long long)a.hs * a.ws;
  const int i = threadIdx.x % kTile;
  if (i >= npix) return;
  for (int q = threadIdx.x / kTile; q * 4 < a.D; q += kProdThreads / kTile) {
    float v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = q * 4 + k < a.D ? __ldg(lg + (q * 4 + k) * plane + i) : -INFINITY;
    *reinterpret_cast<float4 *>(tile + i * stride + q * 4) = make_float4(v[0], v[1], v[2], v[3]);
  }
}

constexpr int kLanes = 8;          // lanes that share a map pixel: a warp normalises four pixels at once

__device__ __forceinline__ float group_max(float v) {
#pragma unroll
  for (int s = kLanes / 2; s > 0; s >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, s));
  return v;
}
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
  for (int s = kLanes / 2; s > 0; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
  return v;
}

// The normalised bins of the CTA's pixel threadIdx.x / kLanes, shared out over its eight lanes: chunk j of a lane are
// the V bins from (sub + 8 j) V on.
template <int V, int NC>
__device__ __forceinline__ void normalised_bins(const float *tile, int stride, const ProdArgs &a, float (&p)[NC][V]) {
  static_assert(kTile * kLanes == kProdThreads, "a pixel per group of lanes");
  const float *row = tile + threadIdx.x / kLanes * stride;
  float mx = -INFINITY;
#pragma unroll
  for (int j = 0; j < NC; ++j) {
    const int d = (threadIdx.x % kLanes + j * kLanes) * V;
#pragma unroll
    for (int k = 0; k < V; ++k) p[j][k] = -INFINITY;
    if (d < a.D) {
      const typename Word<float, V>::type t = *reinterpret_cast<const typename Word<float, V>::type *>(row + d);
      memcpy(p[j], &t, sizeof t);
    }
#pragma unroll
    for (int k = 0; k < V; ++k) mx = fmaxf(mx, p[j][k]);
  }
  if (a.sigmoid) {
#pragma unroll
    for (int j = 0; j < NC; ++j)
#pragma unroll
      for (int k = 0; k < V; ++k) p[j][k] = 1.f / (1.f + expf(-p[j][k]));
    return;
  }
  mx = group_max(mx);
  float sum = 0.f;
#pragma unroll
  for (int j = 0; j < NC; ++j)
#pragma unroll
    for (int k = 0; k < V; ++k) {
      p[j][k] = expf(p[j][k] - mx);
      sum += p[j][k];
    }
  sum = group_sum(sum);
#pragma unroll
  for (int j = 0; j < NC; ++j)
#pragma unroll
    for (int k = 0; k < V; ++k) p[j][k] = __fdiv_rn(p[j][k], sum);
}

// Forward: a CTA owns kTile map pixels, normalises each once and writes the rows of every level pixel that reads one
// of them, from registers.  (A CTA per 32 output rows, which normalised every level pixel anew, took 53 us at
// 6 x 58 x 100 x 64 -> 30 825 rows; this takes 16.5 with the operands in L2, 18.6 cold.)  Bound by instructions and the
// tail, not by memory: issue slots 63 % busy, DRAM 6 % (dist stays in L2), stores 27 % of the path to L2; six CTAs are
// resident on an SM (registers), so that 1392 are 1.57 waves, and the CTA of a map row's last 4 columns takes as long as
// a full one: widths 96, 100, 128 14.5, 16.5, 16.5 us, widths 33 and 64 both 10.4.
template <typename OT, int V, int NC>
__global__ void __launch_bounds__(kProdThreads) dist_from_logits_kernel(const ProdArgs a) {
  extern __shared__ __align__(16) float tile[];
  __shared__ Footprint f;
  const int tiles = (a.ws + kTile - 1) / kTile, b = blockIdx.y, sy = blockIdx.x / tiles;
  const int sx0 = (blockIdx.x - sy * tiles) * kTile, npix = min(kTile, a.ws - sx0);
  const int stride = tile_stride(a.D);
  load_tile(tile, stride, a, a.logits + ((long long)b * a.D * a.hs + sy) * a.ws + sx0, npix);
  stage_footprint(f, a, sy, sx0);
  __syncthreads();
  float p[NC][V];
  normalised_bins<V, NC>(tile, stride, a, p);
  using W = typename Word<OT, V>::type;
  W w[NC];
#pragma unroll
  for (int j = 0; j < NC; ++j) w[j] = pack_bins<OT, V>(p[j]);
  OT *out = reinterpret_cast<OT *>(a.dist) + (long long)b * a.N * a.D + threadIdx.x % kLanes * V;
  const int room = a.D - threadIdx.x % kLanes * V, i = threadIdx.x / kLanes;
  if (i >= npix) return;
  for_each_row(f, a, i, [&](int n) {
    OT *dst = out + (long long)n * a.D;
#pragma unroll
    for (int j = 0; j < NC; ++j)
      if (j * kLanes * V < room) *reinterpret_cast<W *>(dst + j * kLanes * V) = w[j];
  });
}

// Backward: the same ownership.  A pixel's eight lanes sum the incoming gradient over the level pixels that read it, in
// the order of the levels, rows and columns, and form p * (G - <p, G>) (softmax) or p * (1 - p) * G (sigmoid), stored
// along x through shared memory.  (A warp per map pixel, one level pixel after the other: 87 us at the shape above; this
// takes 18.9 with the operands in L2, 25.5 cold.)  Bound by the latency of the gradient's rows (a third of the stalls, the
// barrier behind them another fifth), issue slots (53 % busy) and the same tail; DRAM 27 %.  Widths 96, 100, 128 take 16.8,
// 18.9, 20.6 us, widths 33 and 64 both 12.4.
template <typename GT, int V, int NC>
__global__ void __launch_bounds__(kProdThreads) dist_from_logits_backward_kernel(const ProdArgs a) {
  extern __shared__ __align__(16) float tile[];
  __shared__ Footprint f;
  const int tiles = (a.ws + kTile - 1) / kTile, b = blockIdx.y, sy = blockIdx.x / tiles;
  const int sx0 = (blockIdx.x - sy * tiles) * kTile, npix = min(kTile, a.ws - sx0);
  const int stride = tile_stride(a.D), sub = threadIdx.x % kLanes, pixel = threadIdx.x / kLanes;
  stage_footprint(f, a, sy, sx0);
  load_tile(tile, stride, a, a.logits + ((long long)b * a.D * a.hs + sy) * a.ws + sx0, npix);
  __syncthreads();
  float G[NC][V];
#pragma unroll
  for (int j = 0; j < NC; ++j)
#pragma unroll
    for (int k = 0; k < V; ++k) G[j][k] = 0.f;
  const GT *grad = reinterpret_cast<const GT *>(a.grad_dist) + (long long)b * a.N * a.D + sub * V;
  const int room = a.D - sub * V;
  if (pixel < npix)
    for_each_row(f, a, pixel, [&](int n) {
      const GT *g = grad + (long long)n * a.D;
      float v[NC][V];
#pragma unroll
      for (int j = 0; j < NC; ++j) {
#pragma unroll
        for (int k = 0; k < V; ++k) v[j][k] = 0.f;
        if (j * kLanes * V < room) load_bins<V>(g + j * kLanes * V, v[j]);
      }
#pragma unroll
      for (int j = 0; j < NC; ++j)
#pragma unroll
        for (int k = 0; k < V; ++k) G[j][k] += v[j][k];
    });
  float p[NC][V], pg = 0.f;
  normalised_bins<V, NC>(tile, stride, a, p);
#pragma unroll
  for (int j = 0; j < NC; ++j)
#pragma unroll
    for (int k = 0; k < V; ++k) pg = fmaf(p[j][k], G[j][k], pg);
  pg = group_sum(pg);
  float *row = tile + pixel * stride + sub * V;
#pragma unroll
  for (int j = 0; j < NC; ++j)
    if (j * kLanes * V < room)
#pragma unroll
      for (int k = 0; k < V; ++k)
        row[j * kLanes * V + k] = a.sigmoid ? p[j][k] * (1.f - p[j][k]) * G[j][k] : p[j][k] * (G[j][k] - pg);
  __syncthreads();
  const long long plane = (long long)a.hs * a.ws;
  float *gl = a.grad_logits + ((long long)b * a.D * a.hs + sy) * a.ws + sx0;
  const int i = threadIdx.x % kTile;
  if (i < npix)
    for (int q = threadIdx.x / kTile; q * 4 < a.D; q += kProdThreads / kTile) {
      const float4 t = *reinterpret_cast<const float4 *>(tile + i * stride + q * 4);
      const float v[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (q * 4 + k < a.D) gl[(q * 4 + k) * plane + i] = v[k];
    }
}

size_t tile_bytes(int D) { return (size_t)kTile * tile_stride(D) * sizeof(float); }

// Bins per access: as many as rows start on (D and the tensor's address decide).
int bins_per_access(int D, const void *p, size_t elem) {
  for (int v = 4; v > 1; v /= 2)
    if (D % v == 0 && reinterpret_cast<uintptr_t>(p) % (v * elem) == 0) return v;
  return 1;
}

// NB: bins a lane holds at most, D / 8 rounded up to 8, 16 or 32.
template <typename T, int V, int NB>
cudaError_t launch_typed(const ProdArgs &a, bool backward, dim3 grid, cudaStream_t s) {
  auto kernel = backward ? dist_from_logits_backward_kernel<T, V, NB / V> : dist_from_logits_kernel<T, V, NB / V>;
  kernel<<<grid, kProdThreads, tile_bytes(a.D), s>>>(a);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch(const ProdArgs &a, bool backward, dim3 grid, cudaStream_t s) {
  const int v = bins_per_access(a.D, backward ? a.grad_dist : a.dist, sizeof(T));
#define DFA3D_PRODUCER(V)                                                 \
  (a.D <= 64 ? launch_typed<T, V, 8>(a, backward, grid, s)                \
             : a.D <= 128 ? launch_typed<T, V, 16>(a, backward, grid, s)  \
                          : launch_typed<T, V, 32>(a, backward, grid, s))
  return v == 4 ? DFA3D_PRODUCER(4) : v == 2 ? DFA3D_PRODUCER(2) : DFA3D_PRODUCER(1);
#undef DFA3D_PRODUCER
}

}  // namespace

int dist_producer_max_bins() { return kMaxBins; }

cudaError_t launch_dist_from_logits(const float *logits, const int64_t *shapes, int shape_stride,
                                    const int64_t *lsi, void *dist, int dist_dtype, int B, int D, int hs,
                                    int ws, int N, int L, bool sigmoid, cudaStream_t s) {
  if (B == 0 || N == 0) return cudaSuccess;
  ProdArgs a{};
  a.logits = logits; a.shapes = shapes; a.lsi = lsi; a.dist = dist;
  a.B = B; a.D = D; a.hs = hs; a.ws = ws; a.N = N; a.L = L; a.shape_stride = shape_stride;
  a.sigmoid = sigmoid ? 1 : 0;
  for (int b0 = 0; b0 < B; b0 += 65535) {
    ProdArgs c = a;
    c.logits = logits + (long long)b0 * D * hs * ws;
    c.dist = static_cast<char *>(dist) + (long long)b0 * N * D * (dist_dtype == 0 ? 4 : 2);
    const dim3 grid((unsigned)((ws + kTile - 1) / kTile) * (unsigned)hs, (unsigned)min(65535, B - b0), 1);
    const cudaError_t e = dist_dtype == 3   ? launch<__half>(c, false, grid, s)
                          : dist_dtype == 1 ? launch<__nv_bfloat16>(c, false, grid, s)
                                            : launch<float>(c, false, grid, s);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_dist_from_logits_backward(const float *logits, const int64_t *shapes, int shape_stride,
                                             const int64_t *lsi, const void *grad_dist, int grad_dtype,
                                             float *grad_logits, int B, int D, int hs, int ws, int N,
                                             int L, bool sigmoid, cudaStream_t s) {
  if (B == 0 || hs == 0 || ws == 0) return cudaSuccess;
  ProdArgs a{};
  a.logits = logits; a.shapes = shapes; a.lsi = lsi; a.grad_dist = grad_dist; a.grad_logits = grad_logits;
  a.B = B; a.D = D; a.hs = hs; a.ws = ws; a.N = N; a.L = L; a.shape_stride = shape_stride;
  a.sigmoid = sigmoid ? 1 : 0;
  for (int b0 = 0; b0 < B; b0 += 65535) {
    ProdArgs c = a;
    c.logits = logits + (long long)b0 * D * hs * ws;
    c.grad_logits = grad_logits + (long long)b0 * D * hs * ws;
    c.grad_dist = static_cast<const char *>(grad_dist) + (long long)b0 * N * D * (grad_dtype == 0 ? 4 : 2);
    const dim3 grid((unsigned)((ws + kTile - 1) / kTile) * (unsigned)hs, (unsigned)min(65535, B - b0), 1);
    const cudaError_t e = grad_dtype == 3   ? launch<__half>(c, true, grid, s)
                          : grad_dtype == 1 ? launch<__nv_bfloat16>(c, true, grid, s)
                                            : launch<float>(c, true, grid, s);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace dfa3d
