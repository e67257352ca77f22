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

constexpr int kTile = 32;          // map pixels per CTA, consecutive in memory: they may run over several map rows
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

// adds the bins of a word to V sums
template <int V, typename T>
__device__ __forceinline__ void add_bins(typename Word<T, V>::type w, float (&sum)[V]) {
  T t[V];
  memcpy(t, &w, sizeof w);
#pragma unroll
  for (int i = 0; i < V; ++i) sum[i] += widen(t[i]);
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

// Which level pixels read the CTA's map pixels p0 .. p0 + kTile - 1 (row-major): per level, x[i] is the first column that
// reads pixel i's map column, and y[r] the first row that reads the r-th map row of the tile.
struct Footprint {
  int2 level[kProdLevels];           // width, first row of dist
  int x[kProdLevels][kTile + 1];
  int y[kProdLevels][kTile + 1];
};

__device__ __forceinline__ void stage_footprint(Footprint &f, const ProdArgs &a, int p0, int rows) {
  const int sy0 = p0 / a.ws, each = kTile + 1 + rows + 1;
  for (int t = threadIdx.x; t < a.L * each; t += kProdThreads) {
    const int l = t / each, i = t - l * each;
    const int h = (int)a.shapes[l * a.shape_stride], w = (int)a.shapes[l * a.shape_stride + 1];
    if (i <= kTile) {
      f.x[l][i] = first_at((int)((unsigned)(p0 + i) % (unsigned)a.ws), (float)a.ws / (float)w, w, a.ws);
      if (i == 0) f.level[l] = make_int2(w, (int)a.lsi[l]);
    } else {
      const int r = i - (kTile + 1);
      f.y[l][r] = first_at(sy0 + r, (float)a.hs / (float)h, h, a.hs);
    }
  }
}

// Calls rows(n) with the rows n[0..K) of dist that read map pixel i of the CTA, K at a time and -1 where there is none,
// levels, rows and columns in order.
template <int K, typename F>
__device__ __forceinline__ void for_each_row(const Footprint &f, const ProdArgs &a, int p0, int i, F rows) {
  const int sy = (p0 + i) / a.ws, r = sy - p0 / a.ws;
  const bool last = p0 + i + 1 == (sy + 1) * a.ws;          // the map row's last pixel: up to the level's edge
  for (int l = 0; l < a.L; ++l) {
    const int2 v = f.level[l];
    const int x0 = f.x[l][i], nx = (last ? v.x : f.x[l][i + 1]) - x0;
    if (nx <= 0) continue;
    const int y0 = f.y[l][r], count = (f.y[l][r + 1] - y0) * nx;
    int first = v.y + y0 * v.x + x0, x = 0;
    for (int k = 0; k < count; k += K) {
      int n[K];
#pragma unroll
      for (int u = 0; u < K; ++u) {
        n[u] = k + u < count && (unsigned)(first + x) < (unsigned)a.N ? first + x : -1;
        if (++x == nx) {
          x = 0;
          first += v.x;
        }
      }
      rows(n);
    }
  }
}

// The tile: row i holds the bins of map pixel i, padded to a multiple of four; rows start four words apart modulo 32
// banks, so that 16-byte accesses are free of conflicts both along a row and from row to row.
__host__ __device__ __forceinline__ int padded(int D) { return (D + 3) & ~3; }
__host__ __device__ __forceinline__ int tile_stride(int D) { return (padded(D) + 31) / 32 * 32 + 4; }

// Logits of the CTA's map pixels into the tile (padding: -inf, so that it vanishes in the softmax).  A thread takes
// four bins of one pixel Q times: four loads along the map each, one 16-byte store.  They are asked for first and stored
// after the footprint is worked out, which hides the one behind the other.
template <int Q>
struct TileLoad {
  float v[Q][4];
  __device__ __forceinline__ void ask(const ProdArgs &a, const float *lg, int npix) {
    const long long plane = (long long)a.hs * a.ws;
    const int i = threadIdx.x % kTile;
#pragma unroll
    for (int j = 0; j < Q; ++j)
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int d = (threadIdx.x / kTile + j * (kProdThreads / kTile)) * 4 + k;
        v[j][k] = i < npix && d < a.D ? __ldg(lg + d * plane + i) : -INFINITY;
      }
  }
  __device__ __forceinline__ void store(float *tile, int stride, const ProdArgs &a) const {
#pragma unroll
    for (int j = 0; j < Q; ++j) {
      const int d = (threadIdx.x / kTile + j * (kProdThreads / kTile)) * 4;
      if (d < a.D)
        *reinterpret_cast<float4 *>(tile + threadIdx.x % kTile * stride + d) = make_float4(v[j][0], v[j][1], v[j][2], v[j][3]);
    }
  }
};

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
// of them, from registers.  us, 6 x 58 x 100 maps to 30 825 rows, the operands of three calls in turn: a CTA per 32 output
// rows, which normalised every level pixel anew, 53; tiles that ended with their map row (3 1/8 of them for 100 columns) / this:
// 64 bins 17.9 / 15.0, 118 bins 30.0 / 27.0, 6 x 29 x 50 maps of 64 to 7250 rows 6.3 / 5.3.  Bound by instructions and the tail,
// not by memory: 1092 CTAs of which six are resident on an SM are 1.23 waves; held to 32 registers for eight CTAs 64 bins gain
// a tenth, bf16 loses 7 % and 59 bins 16 %.  More than 128 bins are held to 64 registers, four CTAs instead of three (75 to 80
// registers, which 32 logits a thread at once take): 129 bins 42.8 -> 36.8, bf16 49.6 -> 43.0; 256 bins 48.1 -> 43.7, bf16 33.2 ->
// 30.1 (48 registers 35.9).
template <typename OT, int V, int NC>
__global__ void __launch_bounds__(kProdThreads, V * NC == 32 ? 4 : 0) dist_from_logits_kernel(const ProdArgs a) {
  extern __shared__ __align__(16) float tile[];
  __shared__ Footprint f;
  const int pixels = a.hs * a.ws, b = blockIdx.y, p0 = blockIdx.x * kTile, npix = min(kTile, pixels - p0);
  const int stride = tile_stride(a.D);
  TileLoad<(V * NC + 3) / 4> load;
  load.ask(a, a.logits + (long long)b * a.D * pixels + p0, npix);
  stage_footprint(f, a, p0, (p0 + npix - 1) / a.ws - p0 / a.ws + 1);
  load.store(tile, stride, a);
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
  for_each_row<1>(f, a, p0, i, [&](const int (&n)[1]) {
    if (n[0] < 0) return;
    OT *dst = out + (long long)n[0] * a.D;
#pragma unroll
    for (int j = 0; j < NC; ++j)
      if (j * kLanes * V < room) *reinterpret_cast<W *>(dst + j * kLanes * V) = w[j];
  });
}

// Backward: the same ownership.  A pixel's eight lanes sum the incoming gradient over the level pixels that read it, in
// the order of the levels, rows and columns, and form p * (G - <p, G>) (softmax) or p * (1 - p) * G (sigmoid), stored
// along the map through shared memory.  us as above: a warp per map pixel, one level pixel after the other, 87; tiles that
// ended with their map row / this: 64 bins 23.9 / 21.0, 118 bins 34.8 / 31.1, the 29 x 50 maps 7.1 / 6.3.  Bound by the latency of
// the gradient's rows at the CTAs that the registers leave room for.
template <typename GT, int V, int NC>
__global__ void __launch_bounds__(kProdThreads) dist_from_logits_backward_kernel(const ProdArgs a) {
  extern __shared__ __align__(16) float tile[];
  __shared__ Footprint f;
  const int pixels = a.hs * a.ws, b = blockIdx.y, p0 = blockIdx.x * kTile, npix = min(kTile, pixels - p0);
  const int stride = tile_stride(a.D), sub = threadIdx.x % kLanes, pixel = threadIdx.x / kLanes;
  {
    TileLoad<(V * NC + 3) / 4> load;
    load.ask(a, a.logits + (long long)b * a.D * pixels + p0, npix);
    stage_footprint(f, a, p0, (p0 + npix - 1) / a.ws - p0 / a.ws + 1);
    load.store(tile, stride, a);
  }
  __syncthreads();
  float G[NC][V];
#pragma unroll
  for (int j = 0; j < NC; ++j)
#pragma unroll
    for (int k = 0; k < V; ++k) G[j][k] = 0.f;
  const GT *grad = reinterpret_cast<const GT *>(a.grad_dist) + (long long)b * a.N * a.D + sub * V;
  const int room = a.D - sub * V;
  // Rows asked for at a time, kept as they are stored until they are summed: a second one costs registers, and so CTAs, that few
  // bins cannot spare (118 fp32 bins gain 14 % by it, 64 lose 4 %), nor 65 to 128 16-bit bins in words of
  // one or two, where it takes as many registers as fp32 (bf16, rows widened when they came / kept / kept, one row: 97 bins 42.7
  // / 32.4 / 28.4 us, 118 bins 43.6 / 26.6 / 26.2; of more than 128 two stay ahead: 130 bins 69.5 / 54.7 / 59.1, 255
  // bins 131 / 67 / 68; words of four bins have two, 128 bins 37.5 / 26.0).
  using W = typename Word<GT, V>::type;
  constexpr int K = V * NC <= 8 || (V * NC == 16 && sizeof(GT) == 2 && V < 4) ? 1 : 2;
  if (pixel < npix)
    for_each_row<K>(f, a, p0, pixel, [&](const int (&n)[K]) {
      W w[K][NC];
#pragma unroll
      for (int u = 0; u < K; ++u)
#pragma unroll
        for (int j = 0; j < NC; ++j) {
          memset(&w[u][j], 0, sizeof(W));
          if (n[u] >= 0 && j * kLanes * V < room)
            w[u][j] = __ldg(reinterpret_cast<const W *>(grad + (long long)n[u] * a.D + j * kLanes * V));
        }
#pragma unroll
      for (int u = 0; u < K; ++u)
#pragma unroll
        for (int j = 0; j < NC; ++j) add_bins<V, GT>(w[u][j], G[j]);
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
  float *gl = a.grad_logits + (long long)b * a.D * pixels + p0;
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
    const dim3 grid((unsigned)(((long long)hs * ws + kTile - 1) / kTile), (unsigned)min(65535, B - b0), 1);
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
    const dim3 grid((unsigned)(((long long)hs * ws + kTile - 1) / kTile), (unsigned)min(65535, B - b0), 1);
    const cudaError_t e = grad_dtype == 3   ? launch<__half>(c, true, grid, s)
                          : grad_dtype == 1 ? launch<__nv_bfloat16>(c, true, grid, s)
                                            : launch<float>(c, true, grid, s);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace dfa3d
