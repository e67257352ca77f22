// Per-camera re-batching of BEV queries (sm_100a): which queries each camera sees, packed rows for
// exactly those queries (no padding to the longest camera), and the combination of the per-camera
// results back into BEV order.
//
// Replaces the Python loops, the `nonzero()` host synchronisations and the zero-padded
// (bs, cams, max_len, ...) tensors of SpatialCrossAttention_DFA3D.forward
// (BEVFormer_DFA3D/projects/mmdet3d_plugin/bevformer/modules/spatial_cross_attention.py:700-722 and
// :741-748).  Semantics kept from there: camera i's query list is taken from batch element 0 of
// bev_mask (:703-705), in ascending query order; the divisor of the combination is the number of
// cameras that see the query in the SAME batch element, at least 1 (:745-748).
//
// Packed layout: batch element j, camera i, its r-th visible query sits in row
//   j * T + offsets[i] + r,     T = offsets[cams] = visible (camera, query) pairs of one batch element,
// which is also the order of the operator's "cameras" b = j * cams + i, so op_offsets[b] = j*T +
// offsets[i] is the operator's per-camera query offset table.
#include <cooperative_groups.h>
#include <stdint.h>

#include "dfa3d_b200.h"
#include "dfa3d_launch.h"

namespace dfa3d {
namespace {

constexpr int kPlanThreads = 1024;

// Whether any of the Z entries of mask row `q` is set.
__device__ __forceinline__ bool sees(const uint8_t *mask, long long q, int Z) {
  if (Z == 4 && (reinterpret_cast<uintptr_t>(mask) & 3u) == 0) return __ldg(reinterpret_cast<const uint32_t *>(mask) + q) != 0;
  bool any = false;
  for (int z = 0; z < Z; ++z) any |= mask[q * Z + z] != 0;
  return any;
}

// Exclusive prefix count of `flag` over the CTA (kPlanThreads threads); returns the CTA total in `total`.
__device__ __forceinline__ int block_exclusive_count(bool flag, int &total, int *warp_sums) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned ballot = __ballot_sync(0xffffffffu, flag);
  const int in_warp = __popc(ballot & ((1u << lane) - 1u));
  if (lane == 0) warp_sums[warp] = __popc(ballot);
  __syncthreads();
  int before = 0, all = 0;
  for (int w = 0; w < kPlanThreads / 32; ++w) {
    const int s = warp_sums[w];
    before += w < warp ? s : 0;
    all += s;
  }
  __syncthreads();
  total = all;
  return before + in_warp;
}

// A camera's queries are shared out over a cluster of CTAs in consecutive ranges; a CTA goes over its range 1024 queries
// at a time.  The CTAs' counts meet in distributed shared memory.  (One CTA per camera, two barriers and a scan for every
// 1024 queries, took 46 + 56 us for 6 x 40 000 queries; a thread per consecutive chunk, without them, 10 + 47: its stores
// do not coalesce.  Both kernels like this: 18.6 us back to back, 7.8 + 15.0 cold.)
constexpr int kCluster = 8;

// Queries of this CTA's range that the camera sees.
__device__ __forceinline__ int count_range(const uint8_t *mask, int q0, int q1, int Z, int *warp_sums) {
  int n = 0;
  for (int q = q0 + threadIdx.x; q < q1; q += kPlanThreads) n += sees(mask, q, Z) ? 1 : 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
  if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = n;
  __syncthreads();
  int all = 0;
  for (int w = 0; w < kPlanThreads / 32; ++w) all += warp_sums[w];
  __syncthreads();
  return all;
}

__device__ __forceinline__ void cluster_range(int Q, int &q0, int &q1) {
  const int per = (Q + kCluster - 1) / kCluster;
  q0 = min(Q, (int)(blockIdx.x % kCluster) * per);
  q1 = min(Q, q0 + per);
}

// Cluster i < cams: number of queries camera i sees (batch element 0).  The other clusters: inv_count[j, q] = 1 / max(1,
// number of cameras that see q in batch element j).
__global__ void __cluster_dims__(kCluster, 1, 1) __launch_bounds__(kPlanThreads)
rebatch_count_kernel(const uint8_t *mask, int cams, int bs, int Q, int Z, int32_t *counts, float *inv_count) {
  __shared__ int warp_sums[kPlanThreads / 32];
  __shared__ int mine;
  const int cam = blockIdx.x / kCluster, rank = blockIdx.x % kCluster;
  if (cam >= cams) {
    const long long n = (long long)bs * Q, step = ((long long)gridDim.x - cams * kCluster) * kPlanThreads;
    for (long long t = ((long long)blockIdx.x - cams * kCluster) * kPlanThreads + threadIdx.x; t < n; t += step) {
      int c = 0;
      for (int i = 0; i < cams; ++i) c += sees(mask + (long long)i * n * Z, t, Z) ? 1 : 0;
      inv_count[t] = 1.f / (float)(c < 1 ? 1 : c);
    }
    return;                                          // the whole cluster leaves here
  }
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  int q0, q1;
  cluster_range(Q, q0, q1);
  const int n = count_range(mask + (long long)cam * bs * Q * Z, q0, q1, Z, warp_sums);
  if (threadIdx.x == 0) mine = n;
  cluster.sync();
  if (rank == 0 && threadIdx.x == 0) {
    int all = 0;
    for (int r = 0; r < kCluster; ++r) all += *cluster.map_shared_rank(&mine, r);
    counts[cam] = all;
  }
  cluster.sync();                                    // nobody leaves while its count is still read
}

// One cluster per camera: fills packed_query / packed_camera and the inverse map row_of; the first also writes the offset
// tables.
__global__ void __cluster_dims__(kCluster, 1, 1) __launch_bounds__(kPlanThreads)
rebatch_fill_kernel(const uint8_t *mask, int cams, int bs, int Q, int Z, const int32_t *counts, int32_t *offsets,
                    int32_t *op_offsets, int32_t *packed_query, int32_t *packed_camera, int32_t *row_of) {
  __shared__ int warp_sums[kPlanThreads / 32];
  __shared__ int mine;
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int cam = blockIdx.x / kCluster, rank = blockIdx.x % kCluster;
  const uint8_t *own = mask + (long long)cam * bs * Q * Z;
  int q0, q1;
  cluster_range(Q, q0, q1);
  const int n = count_range(own, q0, q1, Z, warp_sums);
  if (threadIdx.x == 0) mine = n;
  cluster.sync();
  int running = 0;
  for (int r = 0; r < rank; ++r) running += *cluster.map_shared_rank(&mine, r);
  cluster.sync();
  for (int i = 0; i < cam; ++i) running += __ldg(counts + i);
  if (blockIdx.x == 0) {                 // op_offsets[j*cams + i] = j*T + offsets[i]
    int T = 0;
    for (int i = 0; i < cams; ++i) T += __ldg(counts + i);
    for (int b = threadIdx.x; b <= cams * bs; b += kPlanThreads) {
      const int i = b % cams;
      int at = 0;
      for (int c = 0; c < i; ++c) at += __ldg(counts + c);
      op_offsets[b] = b / cams * T + at;
      if (b < cams) offsets[b] = at;
    }
    if (threadIdx.x == 0) offsets[cams] = T;
  }
  for (int base = q0; base < q1; base += kPlanThreads) {
    const int q = base + threadIdx.x;
    const bool f = q < q1 && sees(own, q, Z);
    int total;
    const int pos = running + block_exclusive_count(f, total, warp_sums);
    if (f) { packed_query[pos] = q; packed_camera[pos] = cam; }
    if (q < q1) row_of[(long long)cam * Q + q] = f ? pos : -1;
    running += total;
  }
}

// dst[j*T + p, :] = scale[j, q] * src[cam*cam_stride + j*batch_stride + q, :],  q = packed_query[p],
// cam = packed_camera[p].  VEC = 4: rows of W floats handled as float4 (W % 4 == 0, aligned bases).
template <int VEC>
__global__ void __launch_bounds__(256)
rebatch_gather_kernel(const float *src, const int32_t *packed_query, const int32_t *packed_camera,
                      const int32_t *offsets, int cams, int bs, int Q, int W, long long cam_stride,
                      long long batch_stride, const float *scale, float *dst) {
  const int T = offsets[cams];
  const int wv = W / VEC;
  const long long n = (long long)bs * T * wv;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    const long long row = t / wv;
    const int v = (int)(t - row * wv);
    const int j = (int)(row / T), p = (int)(row - (long long)j * T);
    const int q = packed_query[p], cam = packed_camera[p];
    const float s = scale ? scale[(long long)j * Q + q] : 1.f;
    const float *sp = src + ((long long)cam * cam_stride + (long long)j * batch_stride + q) * W;
    if (VEC == 4) {
      float4 x = __ldg(reinterpret_cast<const float4 *>(sp) + v);
      x.x *= s; x.y *= s; x.z *= s; x.w *= s;
      reinterpret_cast<float4 *>(dst + row * W)[v] = x;
    } else {
      dst[row * W + v] = s * __ldg(sp + v);
    }
  }
}

// dst[j, q, :] = scale[j, q] * sum over cameras i that see q of src[j*T + row_of[i, q], :]
// (every element of dst is written: queries no camera sees get zeros).
// A warp per query: its lanes read the query's row index in 32 cameras at once, and then only the rows there are -- one or
// two of six cameras'.  Bound by HBM.  With a thread per four elements, each of which looked all cameras up after a 64-bit
// division, 40 000 queries of 256 elements took 35 us; like this 18.
template <int VEC>
__global__ void __launch_bounds__(256)
rebatch_combine_kernel(const float *src, const int32_t *row_of, const int32_t *offsets, int cams,
                       int bs, int Q, int W, const float *scale, float *dst) {
  constexpr int U = 2;                            // vectors of a row a lane has in flight
  const int T = offsets[cams];
  const int lane = threadIdx.x & 31, wv = W / VEC;
  const long long rows = (long long)bs * Q;
  for (long long jq = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); jq < rows; jq += (long long)gridDim.x * 8) {
    const long long j = jq / Q;
    const int q = (int)(jq - j * Q);
    const float *sj = src + j * T * W;
    const float s = scale ? __ldg(scale + jq) : 1.f;
    for (int v0 = 0; v0 < wv; v0 += 32 * U) {
      float acc[U][VEC];
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int i = 0; i < VEC; ++i) acc[u][i] = 0.f;
      for (int cam0 = 0; cam0 < cams; cam0 += 32) {
        const int r = cam0 + lane < cams ? __ldg(row_of + (long long)(cam0 + lane) * Q + q) : -1;
        for (unsigned seen = __ballot_sync(0xffffffffu, r >= 0); seen; seen &= seen - 1) {
          const float *row = sj + (long long)__shfl_sync(0xffffffffu, r, __ffs(seen) - 1) * W;
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int v = v0 + u * 32 + lane;
            if (v >= wv) continue;
            if (VEC == 4) {
              const float4 x = __ldg(reinterpret_cast<const float4 *>(row) + v);
              acc[u][0] += x.x; acc[u][1 % VEC] += x.y; acc[u][2 % VEC] += x.z; acc[u][3 % VEC] += x.w;
            } else {
              acc[u][0] += __ldg(row + v);
            }
          }
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int v = v0 + u * 32 + lane;
        if (v >= wv) continue;
        if (VEC == 4)
          reinterpret_cast<float4 *>(dst + jq * W)[v] =
              make_float4(s * acc[u][0], s * acc[u][1 % VEC], s * acc[u][2 % VEC], s * acc[u][3 % VEC]);
        else
          dst[jq * W + v] = s * acc[u][0];
      }
    }
  }
}

unsigned grid_for(long long n, int threads) {
  long long g = (n + threads - 1) / threads;
  const long long cap = 148LL * 16;
  return (unsigned)(g < 1 ? 1 : (g > cap ? cap : g));
}

bool vec4_ok(const void *a, const void *b, int W) {
  return W % 4 == 0 && ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15u) == 0;
}

}  // namespace

cudaError_t launch_rebatch_plan(const uint8_t *mask, int cams, int bs, int Q, int Z, int32_t *counts,
                                int32_t *offsets, int32_t *op_offsets, int32_t *packed_query,
                                int32_t *packed_camera, int32_t *row_of, float *inv_count,
                                cudaStream_t s) {
  const long long per_cluster = (long long)kPlanThreads * kCluster;
  const unsigned inv = (unsigned)min(((long long)bs * Q + per_cluster - 1) / per_cluster, 18LL);
  rebatch_count_kernel<<<(cams + inv) * kCluster, kPlanThreads, 0, s>>>(mask, cams, bs, Q, Z, counts, inv_count);
  rebatch_fill_kernel<<<cams * kCluster, kPlanThreads, 0, s>>>(mask, cams, bs, Q, Z, counts, offsets, op_offsets,
                                                                    packed_query, packed_camera, row_of);
  return cudaGetLastError();
}

cudaError_t launch_rebatch_gather(const float *src, const int32_t *packed_query,
                                  const int32_t *packed_camera, const int32_t *offsets, int cams, int bs,
                                  int Q, int W, long long cam_stride, long long batch_stride,
                                  const float *scale, float *dst, long long rows_bound, cudaStream_t s) {
  if (rows_bound <= 0) return cudaSuccess;
  if (vec4_ok(src, dst, W))
    rebatch_gather_kernel<4><<<grid_for(rows_bound * (W / 4), 256), 256, 0, s>>>(
        src, packed_query, packed_camera, offsets, cams, bs, Q, W, cam_stride, batch_stride, scale, dst);
  else
    rebatch_gather_kernel<1><<<grid_for(rows_bound * W, 256), 256, 0, s>>>(
        src, packed_query, packed_camera, offsets, cams, bs, Q, W, cam_stride, batch_stride, scale, dst);
  return cudaGetLastError();
}

cudaError_t launch_rebatch_combine(const float *src, const int32_t *row_of, const int32_t *offsets,
                                   int cams, int bs, int Q, int W, const float *scale, float *dst,
                                   cudaStream_t s) {
  if ((long long)bs * Q <= 0) return cudaSuccess;
  const unsigned grid = (unsigned)min(((long long)bs * Q + 7) / 8, 1LL << 20);
  if (vec4_ok(src, dst, W))
    rebatch_combine_kernel<4><<<grid, 256, 0, s>>>(src, row_of, offsets, cams, bs, Q, W, scale, dst);
  else
    rebatch_combine_kernel<1><<<grid, 256, 0, s>>>(src, row_of, offsets, cams, bs, Q, W, scale, dst);
  return cudaGetLastError();
}

}  // namespace dfa3d
