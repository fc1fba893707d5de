// clue_scores.cu -- post-processing of clustered points on the GPU: silhouette score
// (clue_silhouette) and cluster centroids (clue_cluster_centroids).
//
// The reference computes the silhouette on the host (include/CLUEstering/utils/detail/scores.hpp:17-99):
// for a point i of a cluster with at least two points, a = mean distance to the other points of
// its cluster, b = the smallest mean distance to the points of another cluster, and
// s_i = (b - a) / max(a, b); silhouette(points) averages s_i over those points.  Cluster sums
// run over the cluster's points in ascending index order (the association map's order), and a
// distance is sqrt(sum over dimensions of (l - r)^2) accumulated from 0 in dimension order.
//
// Here a thread takes one point and a run of whole clusters, so that a cluster's sum runs in exactly
// the reference's order and becomes a mean at the cluster's end: per-point scores are bit-identical
// to a sequential evaluation without contracted multiply-adds.  The smallest mean over the runs does
// not depend on their order.  The work is (clustered points)^2 distances.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <string>

#include "clue_internal.h"

namespace clue_b200 {
namespace {

constexpr int kSilThreads = 128;
constexpr int kSilTile = 256;  // clustered points staged per block step

// Floats per staged point: its coordinates, padded for vector loads.
template <int N>
struct SilRec {
  static constexpr int kFloats = N <= 2 ? N : (N + 3) / 4 * 4;
};

// The clustered points in (cluster, index) order: coordinates as records, and every point's smallest
// other mean, FLT_MAX before k_silhouette (which writes every point's own mean in exactly one run).
template <int N>
__global__ void __launch_bounds__(256) k_sil_gather(int n, const float* __restrict__ coords,
                                                    const int32_t* __restrict__ points, const CsrInfo* info,
                                                    float* __restrict__ rec, uint32_t* __restrict__ other) {
  constexpr int F = SilRec<N>::kFloats;
  const int m = info->n_clustered, stride = gridDim.x * blockDim.x;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < m; p += stride) {
    const int i = points[p];
#pragma unroll
    for (int d = 0; d < F; ++d) rec[(size_t)p * F + d] = d < N ? coords[(size_t)d * n + i] : 0.0f;
    other[p] = __float_as_uint(FLT_MAX);
  }
}

// Means of the clusters that start in the g-th of gridDim.y equal parts of the clustered points, for
// the 128 clustered points of block blockIdx.x.
// Bound by the FP32 pipes (a correctly rounded square root per pair) once enough warps are
// resident: 32k points in 36 clusters leave 1.7 warps per scheduler with one thread per point
// streaming everything, so the clusters are spread over gridDim.y (those 32k 2-D points: 3.96 -> 0.67 ms
// with the allocations of every call and its pageable copies gone as well).
template <int N>
__global__ void __launch_bounds__(kSilThreads) k_silhouette(const int32_t* __restrict__ offsets, const CsrInfo* info,
                                                            const float* __restrict__ rec, float* __restrict__ own_mean,
                                                            uint32_t* __restrict__ other) {
  constexpr int F = SilRec<N>::kFloats;
  __shared__ alignas(16) float s_rec[kSilTile * F];
  const int m = info->n_clustered, nc = (int)info->n_clusters;
  const int p = blockIdx.x * kSilThreads + threadIdx.x;
  if ((int)blockIdx.x * kSilThreads >= m) return;
  // first cluster that starts at or after a position
  auto first_from = [&](int64_t q) {
    int lo = 0, hi = nc;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (offsets[mid] < q)
        lo = mid + 1;
      else
        hi = mid;
    }
    return lo;
  };
  const int c0 = first_from((int64_t)m * blockIdx.y / gridDim.y);
  const int c1 = first_from((int64_t)m * (blockIdx.y + 1) / gridDim.y);
  const int c_end = blockIdx.y + 1 == gridDim.y ? nc : c1;
  if (c0 >= c_end) return;
  float x[N];
#pragma unroll
  for (int d = 0; d < N; ++d) x[d] = rec[(size_t)min(p, m - 1) * F + d];
  float b = FLT_MAX, sum = 0.0f;
  int c = c0, end = offsets[c0 + 1];
  const int q0 = offsets[c0], q1 = offsets[c_end];
  for (int base = q0; base < q1; base += kSilTile) {
    const int cnt = min(kSilTile, q1 - base);
    __syncthreads();
    for (int k = threadIdx.x; k < cnt * F; k += kSilThreads) s_rec[k] = rec[(size_t)base * F + k];
    __syncthreads();
    int k = 0;
    while (k < cnt) {  // one cluster's part of the tile, the same for every thread
      const int stop = min(cnt, end - base);
#pragma unroll 4
      for (; k < stop; ++k) {
        float v[F];
        if constexpr (F == 2) {
          const float2 t = reinterpret_cast<const float2*>(s_rec)[k];
          v[0] = t.x, v[1] = t.y;
        } else if constexpr (F == 1) {
          v[0] = s_rec[k];
        } else {
#pragma unroll
          for (int w = 0; w < F / 4; ++w) {
            const float4 t = reinterpret_cast<const float4*>(s_rec)[k * (F / 4) + w];
            v[4 * w] = t.x, v[4 * w + 1] = t.y, v[4 * w + 2] = t.z, v[4 * w + 3] = t.w;
          }
        }
        float dist = 0.0f;
#pragma unroll
        for (int d = 0; d < N; ++d) {
          const float t = __fsub_rn(x[d], v[d]);
          dist = __fadd_rn(dist, __fmul_rn(t, t));
        }
        // (the point itself adds its distance 0 to its own cluster's sum: the sums are
        // non-negative, so that leaves them as the reference's skip of the point does)
        sum = __fadd_rn(sum, __fsqrt_rn(dist));
      }
      if (base + k == end) {  // the cluster is complete (empty ones in between have no mean)
        const int size = end - offsets[c];
        if (p >= offsets[c] && p < end) {
          own_mean[p] = __fdiv_rn(sum, (float)(size - 1));
        } else {
          const float mean = __fdiv_rn(sum, (float)size);
          b = mean < b ? mean : b;  // std::min(acc, val)
        }
        sum = 0.0f;
        do {
          ++c;
          end = c < c_end ? offsets[c + 1] : INT_MAX;
        } while (c < c_end && end == offsets[c]);
      }
    }
  }
  if (p < m && b < FLT_MAX) atomicMin(other + p, __float_as_uint(b));  // means are not negative
}

// Scores in point order (NaN for points that are not scored), for the caller (optional) and for the
// mean, and which points are scored; nothing after a label out of range (reported by the host).
__global__ void __launch_bounds__(256) k_sil_score(int n, const int32_t* __restrict__ cluster_index,
                                                   const int32_t* __restrict__ offsets,
                                                   const int32_t* __restrict__ points, const CsrInfo* info,
                                                   const float* __restrict__ own_mean,
                                                   const uint32_t* __restrict__ other, float* __restrict__ per_point,
                                                   float* __restrict__ score, uint8_t* __restrict__ scored) {
  if (info->bad) return;
  const int m = info->n_clustered, stride = gridDim.x * blockDim.x;
  const int first = blockIdx.x * blockDim.x + threadIdx.x;
  for (int i = first; i < n; i += stride)
    if (cluster_index[i] < 0 || cluster_index[i] >= n) {
      score[i] = NAN;
      if (per_point) per_point[i] = NAN;
      scored[i] = 0;
    }
  for (int p = first; p < m; p += stride) {
    const int i = points[p], c = cluster_index[i];
    const bool valid = offsets[c + 1] - offsets[c] >= 2;
    const float a = own_mean[p], b = __uint_as_float(other[p]);
    const float v = valid ? __fdiv_rn(__fsub_rn(b, a), a < b ? b : a) : NAN;  // std::max(a, b)
    score[i] = v;
    if (per_point) per_point[i] = v;
    scored[i] = valid ? 1 : 0;
  }
}

template <int N>
void launch_silhouette(int n, const float* coords, const int32_t* cluster_index, const int32_t* offsets,
                       const int32_t* points, const CsrInfo* info, float* rec, float* own_mean, uint32_t* other,
                       float* per_point, float* score, uint8_t* scored, cudaStream_t s) {
  const int blocks = std::max(1, std::min((n + 255) / 256, 148 * 16));
  k_sil_gather<N><<<blocks, 256, 0, s>>>(n, coords, points, info, rec, other);
  // enough parts for four waves of 16 blocks an SM, and no part below 64 points
  const int64_t pb = (n + kSilThreads - 1) / kSilThreads;
  const int64_t parts = std::max<int64_t>(1, std::min<int64_t>({(int64_t)148 * 64 / pb, (int64_t)n / 64, 65535}));
  k_silhouette<N><<<dim3((unsigned)pb, (unsigned)parts), kSilThreads, 0, s>>>(offsets, info, rec, own_mean, other);
  k_sil_score<<<blocks, 256, 0, s>>>(n, cluster_index, offsets, points, info, own_mean, other, per_point, score,
                                     scored);
}

constexpr int kCenThreads = 128;

// Centroid of a cluster (reference utils/detail/cluster_centroid.hpp:39-65): in every dimension the
// coordinates summed from 0 in ascending point order (the CSR of clue_get_clusters lists a
// cluster's points that way) with separately rounded FP32 adds, divided by the size as a float: the
// bits of the reference's host loop.  One block per cluster: all threads gather the next 128 points
// while thread d adds up dimension d of the 128 before, so the sum's chain of additions and not the
// gathers' latency bounds it (1M 2-D points in 1000 clusters: 18 us; the whole call and a
// clue_get_clusters before it 9.0 -> 0.21 ms with the absent keys' offsets written in parallel).
__global__ void __launch_bounds__(kCenThreads) k_centroids(int ndim, int n, int capacity,
                                                           const float* __restrict__ coords,
                                                           const int32_t* __restrict__ offsets,
                                                           const int32_t* __restrict__ points, const CsrInfo* info,
                                                           float* __restrict__ centroids, int32_t* __restrict__ sizes) {
  __shared__ float4 s_x[2][kMaxDim][kCenThreads / 4];
  const int nc = (int)info->n_clusters;
  if (nc > capacity || info->bad) return;  // reported by the host
  for (int c = blockIdx.x; c < nc; c += gridDim.x) {
    const int b = offsets[c], e = offsets[c + 1];
    float acc = 0.0f;
    int buf = 0;
    for (int base = b; base < e; base += kCenThreads, buf ^= 1) {
      const int q = base + (int)threadIdx.x;
      if (q < e) {
        const int i = points[q];
        for (int d = 0; d < ndim; ++d) reinterpret_cast<float*>(s_x[buf][d])[threadIdx.x] = coords[(size_t)d * n + i];
      }
      __syncthreads();  // (the buffer written next was summed before this barrier)
      if ((int)threadIdx.x < ndim) {
        const float4* v = s_x[buf][threadIdx.x];
        const int cnt = min(kCenThreads, e - base);
        int k = 0;
        for (; k + 4 <= cnt; k += 4) {
          const float4 t = v[k >> 2];
          acc = fadd(fadd(fadd(fadd(acc, t.x), t.y), t.z), t.w);
        }
        for (; k < cnt; ++k) acc = fadd(acc, reinterpret_cast<const float*>(v)[k]);
      }
    }
    if ((int)threadIdx.x < ndim) centroids[(size_t)c * ndim + threadIdx.x] = fdiv(acc, (float)(e - b));
    if (sizes && threadIdx.x == 0) sizes[c] = e - b;
    __syncthreads();  // the next cluster starts with the first buffer
  }
}

size_t up256(size_t x) { return (x + 255) / 256 * 256; }

}  // namespace
}  // namespace clue_b200

using namespace clue_b200;

extern "C" {

clue_status clue_cluster_centroids(clue_context ctx, int32_t ndim, int32_t n, const float* coords,
                                   const int32_t* cluster_index, int32_t capacity, float* centroids,
                                   int32_t* sizes, int32_t* n_clusters_out, void* stream) {
  if (!ctx || !coords || !cluster_index || (!centroids && capacity > 0) || n <= 0 || capacity < 0 || ndim < 1 ||
      ndim > kMaxDim) {
    set_error("clue_cluster_centroids: null argument, n <= 0, capacity < 0 or ndim outside [1, 10]");
    return CLUE_ERR_INVALID_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  Workspace& ws = context_workspace(ctx);
  const size_t off_bytes = up256(((size_t)n + 1) * 4);
  clue_status st = post_reserve(ws, 256 + off_bytes + (size_t)n * 4, sizeof(CsrInfo));
  if (st != CLUE_OK) return st;
  char* base = static_cast<char*>(ws.post);
  CsrInfo* info = reinterpret_cast<CsrInfo*>(base);
  int32_t* offsets = reinterpret_cast<int32_t*>(base + 256);
  int32_t* points = reinterpret_cast<int32_t*>(base + 256 + off_bytes);
  int prev = 0;
  cudaGetDevice(&prev);
  cudaSetDevice(ws.device);
  const bool was_busy = ws.busy;
  st = clusters_csr(ws, n, cluster_index, offsets, points, info, s);
  cudaError_t e = cudaSuccess;
  if (st == CLUE_OK) {
    if (capacity > 0) {
      k_centroids<<<std::min(capacity, 148 * 16), kCenThreads, 0, s>>>(ndim, n, capacity, coords, offsets, points, info,
                                                                       centroids, sizes);
      ++ws.launches;
    }
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(ws.post_host, info, sizeof(CsrInfo), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  }
  cudaSetDevice(prev);
  if (st != CLUE_OK) return st;
  if (e != cudaSuccess) {
    set_error(std::string("clue_cluster_centroids: ") + cudaGetErrorString(e));
    return CLUE_ERR_CUDA;
  }
  ws.busy = was_busy;  // all of it was waited for
  const CsrInfo* h = static_cast<const CsrInfo*>(ws.post_host);
  if (h->bad) {
    set_error("clue_get_clusters: cluster index outside [-1, n)");
    return CLUE_ERR_OUT_OF_RANGE;
  }
  if (n_clusters_out) *n_clusters_out = (int32_t)h->n_clusters;
  if ((int64_t)h->n_clusters > capacity) {
    set_error("clue_cluster_centroids: more clusters (" + std::to_string(h->n_clusters) + ") than the capacity (" +
              std::to_string(capacity) + ")");
    return CLUE_ERR_CAPACITY;
  }
  return CLUE_OK;
}

clue_status clue_silhouette(clue_context ctx, int32_t ndim, int32_t n, const float* coords,
                            const int32_t* cluster_index, float* per_point, float* mean, void* stream) {
  if (!ctx || !coords || !cluster_index || n <= 0 || ndim < 1 || ndim > kMaxDim) {
    set_error("clue_silhouette: null argument, n <= 0 or ndim outside [1, 10]");
    return CLUE_ERR_INVALID_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  Workspace& ws = context_workspace(ctx);
  const size_t nn = (size_t)n, rec_floats = ndim <= 2 ? (size_t)ndim : (size_t)(ndim + 3) / 4 * 4;
  // info, then the scores and which points are scored (read back in one copy), then the rest
  const size_t o_score = 256, o_scored = o_score + nn * 4, o_off = up256(o_scored + nn), o_pts = o_off + up256((nn + 1) * 4),
               o_rec = o_pts + up256(nn * 4), o_own = o_rec + up256(nn * rec_floats * 4), o_other = o_own + up256(nn * 4),
               total = o_other + up256(nn * 4);
  const size_t back = mean ? o_scored + nn : sizeof(CsrInfo);
  clue_status st = post_reserve(ws, total, back);
  if (st != CLUE_OK) return st;
  char* base = static_cast<char*>(ws.post);
  CsrInfo* info = reinterpret_cast<CsrInfo*>(base);
  float* score = reinterpret_cast<float*>(base + o_score);
  uint8_t* scored = reinterpret_cast<uint8_t*>(base + o_scored);
  int32_t* offsets = reinterpret_cast<int32_t*>(base + o_off);
  int32_t* points = reinterpret_cast<int32_t*>(base + o_pts);
  float* rec = reinterpret_cast<float*>(base + o_rec);
  float* own_mean = reinterpret_cast<float*>(base + o_own);
  uint32_t* other = reinterpret_cast<uint32_t*>(base + o_other);
  int prev = 0;
  cudaGetDevice(&prev);
  cudaSetDevice(ws.device);
  const bool was_busy = ws.busy;
  st = clusters_csr(ws, n, cluster_index, offsets, points, info, s);
  cudaError_t e = cudaSuccess;
  if (st == CLUE_OK) {
#define CLUE_SIL(N)                                                                                              \
  case N:                                                                                                        \
    launch_silhouette<N>(n, coords, cluster_index, offsets, points, info, rec, own_mean, other, per_point,       \
                         score, scored, s);                                                                      \
    break;
    switch (ndim) {
      CLUE_SIL(1) CLUE_SIL(2) CLUE_SIL(3) CLUE_SIL(4) CLUE_SIL(5) CLUE_SIL(6) CLUE_SIL(7) CLUE_SIL(8) CLUE_SIL(9)
      default: launch_silhouette<10>(n, coords, cluster_index, offsets, points, info, rec, own_mean, other, per_point,
                                     score, scored, s);
    }
#undef CLUE_SIL
    ws.launches += 3;
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(ws.post_host, base, back, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  }
  cudaSetDevice(prev);
  if (st != CLUE_OK) return st;
  if (e != cudaSuccess) {
    set_error(std::string("clue_silhouette: ") + cudaGetErrorString(e));
    return CLUE_ERR_CUDA;
  }
  ws.busy = was_busy;  // all of it was waited for
  if (static_cast<const CsrInfo*>(ws.post_host)->bad) {
    set_error("clue_get_clusters: cluster index outside [-1, n)");
    return CLUE_ERR_OUT_OF_RANGE;
  }
  if (mean) {
    // the average in index order over the points of clusters with at least two points, in
    // FP32 like the reference's reduce
    const float* h = reinterpret_cast<const float*>(static_cast<const char*>(ws.post_host) + o_score);
    const uint8_t* ok = reinterpret_cast<const uint8_t*>(static_cast<const char*>(ws.post_host) + o_scored);
    float acc = 0.0f;
    int64_t cnt = 0;
    for (int i = 0; i < n; ++i) {
      if (!ok[i]) continue;
      acc += h[i];
      ++cnt;
    }
    *mean = acc / (float)cnt;
  }
  return CLUE_OK;
}

}  // extern "C"
