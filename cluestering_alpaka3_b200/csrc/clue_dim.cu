// clue_dim.cu -- the five CLUE stages for points of CLUE_NDIM dimensions.
//
// Compiled once per dimensionality (-DCLUE_NDIM=1..10) so the templates of one
// dimension build in parallel.  Stage map against the reference's serial path
// (include/CLUEstering/core/detail/Clusterer.hpp:134-171):
//   k_bbox_* / k_grid    compute_tile_size        core/detail/ComputeTiles.hpp:13-27
//   k_bin + radix sort   Tiles::fill              data_structures/internal/Tiles.hpp:92-96
//   (k_bin_composite)    (one (tile, Morton) sort on the symmetric density path)
//   k_density            KernelCalculateLocalDensity  core/detail/ClusteringKernels.hpp:66-107
//   k_density_sym /      the same sums in spatial order (exponential / Gaussian kernels):
//   k_density_spatial    symmetric pair sweep or one-sided sweep over Morton blocks
//   k_nearest_higher     KernelCalculateNearestHigher core/detail/ClusteringKernels.hpp:109-212
//                        and KernelFindClusters   core/detail/ClusteringKernels.hpp:214-244
//   k_seed_labels, k_labels (k_jump)  Followers::fill + KernelAssignClusters
//                        data_structures/internal/Followers.hpp:27-30,
//                        core/detail/ClusteringKernels.hpp:246-281
//
// One call clusters E independent events (E = 1 for a plain make_clusters).  Event e owns
// points [pt_base, pt_base + pt_count) and global tiles [tile_base, tile_base + ntiles) of its
// own reference grid; tile keys are event-major, so one stable sort of (tile, index) pairs
// orders every event by tile while keeping events contiguous.
//
// Layout in HBM: points are reordered by tile into float4 records {coords..., payload}: by
// ascending index inside a tile for the reference-order density, by Morton code inside a tile
// for the spatial sweeps.  A CTA processes a chunk of 128 home points of one tile (four warps
// of 32).  The reference-order density reads whole candidate tiles and sums what lies within reach
// of the warp's homes; the spatial sweeps take one 32-record Morton block at a time, skip blocks
// whose bounding box is out of reach, and read the candidates from shared memory (nearest higher) or,
// as neighbouring pairs, from a shared-memory copy by component (symmetric density).
#include <atomic>
#include <cstdlib>
#include <cstring>

#include "clue_internal.h"

#ifndef CLUE_NDIM
#error "CLUE_NDIM must be defined"
#endif

namespace clue_b200 {
namespace {

constexpr int kTileThreads = 128;
constexpr int kChunkWarps = kTileThreads / 32;
constexpr int kChunk = kChunkPoints;  // home points per CTA in the density / nearest-higher sweeps
static_assert(kChunkPoints == kTileThreads, "one home point per thread");
struct InPtrs {
  const float* c[kMaxDim];
  const float* w;
};

// Event tables of one call.
struct Events {
  EvGrid* eg;               // [E]
  const int32_t* pt;        // [E + 1] point offsets
  const int32_t* tile;      // [E + 1] global tile offsets
  const int32_t* chunk_ev;  // [n / 1024 + 1] event of the first point of every 1024-point chunk
};
constexpr int kEvChunkShift = 10;

// What the nearest-higher search hands to the label stage.
struct SeedBufs {
  int32_t* par;    // label parents: the nearest higher, -1 for seeds and points without one
  int32_t* nh;     // nearest highers, or null
  uint32_t* bits;  // seeds, one bit per point in original order
  int32_t* list;   // seeds' positions
};

// The lane's number, read once: left to itself the compiler reads the special register again at
// every use in a long kernel.
__device__ __forceinline__ int lane_id() {
  int lane = threadIdx.x & 31;
  asm volatile("" : "+r"(lane));
  return lane;
}

// Warp-wide minima and maxima, one instruction each (redux.sync; the float forms are sm_100a).
__device__ __forceinline__ int warp_min_i(int v) { return __reduce_min_sync(0xffffffffu, v); }
__device__ __forceinline__ int warp_max_i(int v) { return __reduce_max_sync(0xffffffffu, v); }
__device__ __forceinline__ uint32_t warp_min_u(uint32_t v) { return __reduce_min_sync(0xffffffffu, v); }
__device__ __forceinline__ uint32_t warp_max_u(uint32_t v) { return __reduce_max_sync(0xffffffffu, v); }
__device__ __forceinline__ float warp_min_f(float v) {
  float r;
  asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float warp_max_f(float v) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}

// Entry p of an order; a null order is the identity.
__device__ __forceinline__ int order_at(const int32_t* __restrict__ order, int p) {
  return order ? __ldg(order + p) : p;
}

// Largest e in [0, E) with base[e] <= x.
__device__ __forceinline__ int find_event(const int32_t* __restrict__ base, int E, int x) {
  int lo = 0, hi = E - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(base + mid) <= x)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

template <int N>
__device__ __forceinline__ void load_rec(const float4* __restrict__ rec, int pos, float* x, float& payload) {
  constexpr int W = Rec<N>::kWords;
  float buf[4 * W];
#pragma unroll
  for (int k = 0; k < W; ++k) {
    const float4 v = __ldg(rec + (size_t)pos * W + k);
    buf[4 * k + 0] = v.x;
    buf[4 * k + 1] = v.y;
    buf[4 * k + 2] = v.z;
    buf[4 * k + 3] = v.w;
  }
#pragma unroll
  for (int d = 0; d < N; ++d) x[d] = buf[d];
  payload = buf[Rec<N>::kPayload];
}

template <int N>
__device__ __forceinline__ void store_rec(float4* __restrict__ rec, int pos, const float* x, float payload) {
  constexpr int W = Rec<N>::kWords;
  float buf[4 * W];
#pragma unroll
  for (int k = 0; k < 4 * W; ++k) buf[k] = 0.0f;
#pragma unroll
  for (int d = 0; d < N; ++d) buf[d] = x[d];
  buf[Rec<N>::kPayload] = payload;
#pragma unroll
  for (int k = 0; k < W; ++k)
    rec[(size_t)pos * W + k] = make_float4(buf[4 * k], buf[4 * k + 1], buf[4 * k + 2], buf[4 * k + 3]);
}

// Search box of one point in "virtual" bins: the reference's [getBin(x - r), getBin(x + r)]
// (TilesView.hpp:72-82, wrapped boxes extended by nperdim), shifted down by nperdim when a
// wrapped box starts above the home bin, so that every lane of a warp expresses its box
// in the same frame around the home tile.  The tile of virtual bin v is v mod nperdim.
template <int N>
__device__ __forceinline__ void lane_box(const KParams& kp, const EvGrid* __restrict__ g, const float* x,
                                         float r, const int* hb, int* lo, int* hi) {
  const int npd = g->nperdim;
#pragma unroll
  for (int d = 0; d < N; ++d) {
    const bool wr = kp.wrapped[d] != 0;
    int a = get_bin(fsub(x[d], r), g->mn[d], g->mx[d], g->size[d], wr, npd);
    int b = get_bin(fadd(x[d], r), g->mn[d], g->mx[d], g->size[d], wr, npd);
    if (wr && a > b) b += npd;
    if (wr && a > hb[d]) {
      a -= npd;
      b -= npd;
    }
    lo[d] = a;
    hi[d] = b;
  }
}

template <int N>
__device__ __forceinline__ void home_bins(const EvGrid* __restrict__ g, int t, int* hb) {
  const int lt = t - g->tile_base;
#pragma unroll
  for (int d = 0; d < N; ++d) hb[d] = (lt / g->stride[d]) % g->nperdim;
}

// Tile bin of virtual bin v: lane_box keeps v within one period of the grid, [-npd, 2 npd).
__device__ __forceinline__ int wrap_bin(int v, int npd) { return v < 0 ? v + npd : (v >= npd ? v - npd : v); }

// Box of one warp's 32 records (lanes past the end repeat a record of the block): lo[N],
// hi[N] and the largest payload, written as block b.
template <int N>
__device__ __forceinline__ void write_block_box(float4* __restrict__ blk, int b, const float* x, float pl) {
  constexpr int BW = Blk<N>::kWords;
  const int lane = threadIdx.x & 31;
  float out[4 * BW];
#pragma unroll
  for (int k = 0; k < 4 * BW; ++k) out[k] = 0.0f;
#pragma unroll
  for (int d = 0; d < N; ++d) {
    out[d] = warp_min_f(x[d]);
    out[N + d] = warp_max_f(x[d]);
  }
  out[2 * N] = warp_max_f(pl);
  if (lane < BW) {
    float4 v;
#pragma unroll
    for (int k = 0; k < BW; ++k)
      if (k == lane) v = make_float4(out[4 * k], out[4 * k + 1], out[4 * k + 2], out[4 * k + 3]);
    blk[(size_t)b * BW + lane] = v;
  }
}

template <int N>
__device__ __forceinline__ void load_box(const float4* __restrict__ a, int i, float* bb) {
  constexpr int BW = Blk<N>::kWords;
#pragma unroll
  for (int k = 0; k < BW; ++k) {
    const float4 t4 = __ldg(a + (size_t)i * BW + k);
    bb[4 * k] = t4.x;
    bb[4 * k + 1] = t4.y;
    bb[4 * k + 2] = t4.z;
    bb[4 * k + 3] = t4.w;
  }
}

// A block of up to 32 consecutive records staged in the warp's shared-memory slot: lane k
// copies record p0 + k; smem_rec() then reads record j with broadcast loads (every lane reads
// the same address), one 16-byte load per record word.
// With sq / mq given, the records' tile-sorted positions mq[p0 + k] are staged in sq as well.
template <int N>
__device__ __forceinline__ void stage_block(float4* sm, const float4* __restrict__ rec, int p0, int cnt,
                                            int32_t* sq = nullptr, const int32_t* __restrict__ mq = nullptr) {
  constexpr int W = Rec<N>::kWords;
  const int lane = threadIdx.x & 31;
  __syncwarp();  // the previous block's readers are done
  if (lane < cnt) {
#pragma unroll
    for (int k = 0; k < W; ++k) sm[lane * W + k] = __ldg(rec + (size_t)(p0 + lane) * W + k);
    if (sq) sq[lane] = order_at(mq, p0 + lane);
  }
  __syncwarp();
}
template <int N>
__device__ __forceinline__ void smem_rec(const float4* sm, int j, float* c, float& payload) {
  constexpr int W = Rec<N>::kWords;
  float r[4 * W];
#pragma unroll
  for (int k = 0; k < W; ++k) {
    const float4 v = sm[j * W + k];
    r[4 * k] = v.x;
    r[4 * k + 1] = v.y;
    r[4 * k + 2] = v.z;
    r[4 * k + 3] = v.w;
  }
#pragma unroll
  for (int d = 0; d < N; ++d) c[d] = r[d];
  payload = r[Rec<N>::kPayload];
}

// Tiles of the union box [wl, wh] of a warp's search boxes, lane l's tile v (in_batch: whether it has
// one) looked up by all lanes at once; f(v, rank, pb, pe) gets the non-empty ones in lane order with
// their records [pb, pe).  rank is the tile's lexicographic position in the union, so it orders two
// tiles of a lane's box as the reference's iteration does.
template <int N, class F>
__device__ __forceinline__ void batch_tiles(const EvGrid* __restrict__ g, const int32_t* __restrict__ off,
                                            const int* wl, const int* wh, const int* v, bool in_batch, F&& f) {
  int u = g->tile_base, rank = 0;
#pragma unroll
  for (int d = 0; d < N; ++d) {
    u += g->stride[d] * wrap_bin(v[d], g->nperdim);
    rank = rank * (wh[d] - wl[d] + 1) + (v[d] - wl[d]);
  }
  int pb = 0, pe = 0;
  if (in_batch) {
    pb = off[u];
    pe = off[u + 1];
  }
  for (unsigned m = __ballot_sync(0xffffffffu, pb < pe); m; m &= m - 1) {
    const int src = __ffs(m) - 1;
    int tv[N];
#pragma unroll
    for (int d = 0; d < N; ++d) tv[d] = __shfl_sync(0xffffffffu, v[d], src);
    f(tv, __shfl_sync(0xffffffffu, rank, src), __shfl_sync(0xffffffffu, pb, src), __shfl_sync(0xffffffffu, pe, src));
  }
}

// All tiles of the union box more than done_ring tiles away from the home tile, lexicographically.
template <int N, class F>
__device__ __forceinline__ void box_tiles(const EvGrid* __restrict__ g, const int32_t* __restrict__ off,
                                          const int* hb, const int* wl, const int* wh, int done_ring, int lane,
                                          F&& f) {
  int64_t total = 1;
#pragma unroll
  for (int d = 0; d < N; ++d) total *= wh[d] - wl[d] + 1;
  for (int64_t base = 0; base < total; base += 32) {
    int64_t id = base + lane;
    const bool in = id < total;
    int v[N], ring = 0;
#pragma unroll
    for (int d = N - 1; d >= 0; --d) {
      const int ext = wh[d] - wl[d] + 1;
      if (d == 0) {
        v[d] = wl[d] + (int)(in ? id : 0);
      } else if (total <= INT_MAX) {
        v[d] = wl[d] + (int)((uint32_t)id % (uint32_t)ext);
        id = (uint32_t)id / (uint32_t)ext;
      } else {
        v[d] = wl[d] + (int)(id % ext);
        id /= ext;
      }
      ring = max(ring, abs(v[d] - hb[d]));
    }
    batch_tiles<N>(g, off, wl, wh, v, in && ring > done_ring, f);
  }
}

// Spatial sweep of one warp over the Morton-ordered records of its search-box tiles: the own tile
// first, then the union of the warp's boxes.  vis(p0, p1, need, rank) gets every 32-record block that
// some lane may need: the lane's box holds the tile, the block's box lower bound is within bound()
// and its largest payload reaches pmin.  rank: see batch_tiles.
//
// The tests are bound by instruction issue, so they are spread over the lanes: lane l looks up
// tile l of the union (32 at a time) and tests block l of a super-block (1024 records) against the
// warp's box, its largest bound and its smallest pmin; only blocks that pass get the test of every
// lane against its own point.  (Testing every block by every lane took 30 tests of about 30
// instructions per warp of the calorimeter batch's nearest-higher search, where 7.6 blocks are
// visited.)
//
// With NEAREST, p_home is the lane's own Morton position: the blocks of the warp's own positions
// come first, then the blocks of a super-block in the order of their distance from the warp's
// box, and (up to three dimensions) the tiles next to the home tile before the others, so that
// bound() shrinks early.  Without it every tile's blocks are visited in Morton order, so
// order-sensitive sums do not depend on how records are aligned to blocks (a batch and a single
// event give identical results).
template <int N, class M, bool NEAREST, class Bound, class Visit>
__device__ __forceinline__ void spatial_sweep(const KParams& kp, const EvGrid* __restrict__ g,
                                              const int32_t* __restrict__ off, const int* hb, const int* lo,
                                              const int* hi, bool valid, const float* x,
                                              const float4* __restrict__ blk, const float4* __restrict__ sblk,
                                              float pmin, int p_home, Bound&& bound, Visit&& vis) {
  constexpr int BW = Blk<N>::kWords;
  const int lane = lane_id();
  const int ph_lo = NEAREST ? warp_min_i(valid ? p_home : INT_MAX) : 0;
  const int ph_hi = NEAREST ? warp_max_i(valid ? p_home : INT_MIN) : 0;
  int wl[N], wh[N];
  float hlo[N], hhi[N];  // box of the warp's own points
#pragma unroll
  for (int d = 0; d < N; ++d) {
    wl[d] = warp_min_i(valid ? lo[d] : INT_MAX);
    wh[d] = warp_max_i(valid ? hi[d] : INT_MIN);
    hlo[d] = warp_min_f(valid ? x[d] : INFINITY);
    hhi[d] = warp_max_f(valid ? x[d] : -INFINITY);
  }
  // one non-empty tile [pb, pe): its super-blocks and blocks that some lane may need
  auto visit_tile = [&](const int* v, int rank, int pb, int pe, bool home_tile) {
    bool inbox = valid;
#pragma unroll
    for (int d = 0; d < N; ++d) inbox = inbox && v[d] >= lo[d] && v[d] <= hi[d];
    if (!__any_sync(0xffffffffu, inbox)) return;
    const float rmin = warp_min_f(inbox ? pmin : INFINITY);
    const int bf = pb >> 5, bl = (pe - 1) >> 5;
    const int sf = bf >> 5, ns = (bl >> 5) - sf + 1;
    int s = NEAREST && home_tile ? ph_lo >> 10 : sf;  // the super-block of the own points first
    for (int k = 0; k < ns; ++k, s = s + 1 == sf + ns ? sf : s + 1) {
      const float bmax = warp_max_f(inbox ? bound() : -INFINITY);
      if (kp.lb_ok && ns > 1) {
        float bb[4 * BW];
        load_box<N>(sblk, s, bb);
        if (!(lower_box<N, M>(hlo, hhi, bb, bb + N, kp.mpar) <= bmax && bb[2 * N] >= rmin)) continue;
      }
      const int bi = (s << 5) + lane;
      bool c = bi >= bf && bi <= bl;
      float lb = 0.0f;
      if (kp.lb_ok && c) {
        float bb[4 * BW];
        load_box<N>(blk, bi, bb);
        lb = lower_box<N, M>(hlo, hhi, bb, bb + N, kp.mpar);
        c = lb <= bmax && bb[2 * N] >= rmin;
      }
      if (NEAREST && home_tile && bi >= ph_lo >> 5 && bi <= ph_hi >> 5) lb = -1.0f;
      unsigned mask = __ballot_sync(0xffffffffu, c);
      while (mask) {
        int src;
        if (NEAREST) {
          const float near = warp_min_f(c ? lb : INFINITY);
          if (kp.lb_ok && near > warp_max_f(inbox ? bound() : -INFINITY)) break;  // so are the rest
          src = __ffs(__ballot_sync(0xffffffffu, c && lb == near)) - 1;
          c = c && lane != src;
          mask &= ~(1u << src);
        } else {
          src = __ffs(mask) - 1;
          mask &= mask - 1;
        }
        const int b = (s << 5) + src;
        bool need = inbox;
        if (kp.lb_ok) {
          float bb[4 * BW];
          load_box<N>(blk, b, bb);
          need = need && lower_point<N, M>(x, bb, bb + N, kp.mpar) <= bound() && bb[2 * N] >= pmin;
        }
        if (__any_sync(0xffffffffu, need)) vis(max(pb, b << 5), min(pe, (b + 1) << 5), need, rank);
      }
    }
  };
  batch_tiles<N>(g, off, wl, wh, hb, lane == 0, [&](const int* v, int rank, int pb, int pe) {
    visit_tile(v, rank, pb, pe, true);
  });
  auto other = [&](const int* v, int rank, int pb, int pe) { visit_tile(v, rank, pb, pe, false); };
  int done_ring = 0;  // tiles up to this ring around the home tile are done
  if (NEAREST && N <= 3) {
    int v[N], id = lane;
    bool in = true, home = true;
#pragma unroll
    for (int d = N - 1; d >= 0; --d) {
      v[d] = hb[d] - 1 + id % 3;
      id /= 3;
      in = in && v[d] >= wl[d] && v[d] <= wh[d];
      home = home && v[d] == hb[d];
    }
    batch_tiles<N>(g, off, wl, wh, v, in && id == 0 && !home, other);
    done_ring = 1;
  }
  bool rest = false;
#pragma unroll
  for (int d = 0; d < N; ++d) rest = rest || hb[d] - wl[d] > done_ring || wh[d] - hb[d] > done_ring;
  if (rest) box_tiles<N>(g, off, hb, wl, wh, done_ring, lane, other);
}

// ---- stage 1: bounding box, grid, bins --------------------------------------

// Resets the per-call state; for a plain call also writes the event table of its one event.
template <int N>
__global__ void k_init(const KParams kp, Events ev, int32_t* ev_pt, int32_t* ev_tile, uint32_t* seed_bits,
                       uint32_t* chunk_total, DevStatus* st) {
  if (blockIdx.x == 0) {
    uint32_t* s = reinterpret_cast<uint32_t*>(st);
    for (int k = threadIdx.x; k < (int)(sizeof(DevStatus) / 4); k += blockDim.x) s[k] = 0u;
    if (chunk_total && threadIdx.x == 0) *chunk_total = (uint32_t)(kp.n / kChunk + kp.ntiles + 1);
  }
  const int stride = gridDim.x * blockDim.x;
  for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < (kp.n + 31) / 32; w += stride) seed_bits[w] = 0u;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < kp.n_events; e += stride) {
    EvGrid& g = ev.eg[e];
    for (int d = 0; d < kMaxDim; ++d) {
      g.enc_min[d] = 0xffffffffu;
      g.enc_max[d] = 0u;
    }
    g.seed_candidates = 0;
    g.wmax_bits = 0u;
    if (kp.n_events == 1) {
      g.nperdim = kp.nperdim0;
      g.ntiles = kp.ntiles;
      g.tile_base = 0;
      g.pt_base = 0;
      g.pt_count = kp.n;
      for (int d = 0; d < kMaxDim; ++d) g.stride[d] = kp.stride0[d];
      ev_pt[0] = 0;
      ev_pt[1] = kp.n;
      ev_tile[0] = 0;
      ev_tile[1] = kp.ntiles;
    }
  }
}

// Bounding box and largest |weight| of a single event: per-thread, warp and block reductions,
// then one set of atomics per CTA.
template <int N>
__global__ void __launch_bounds__(256) k_bbox_single(InPtrs in, int n, EvGrid* g, DevStatus* st) {
  uint32_t emn[N], emx[N];
#pragma unroll
  for (int d = 0; d < N; ++d) {
    emn[d] = 0xffffffffu;
    emx[d] = 0u;
  }
  bool bad = false;
  uint32_t wmax = 0u;
  auto take = [&](const float* x, float w) {
#pragma unroll
    for (int d = 0; d < N; ++d) {
      bad |= !isfinite(x[d]);
      const uint32_t e = enc_float(x[d]);
      emn[d] = min(emn[d], e);
      emx[d] = max(emx[d], e);
    }
    bad |= !isfinite(w);
    wmax = max(wmax, __float_as_uint(fabsf(w)));
  };
  const int stride = gridDim.x * blockDim.x;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  // four points per thread and step, their loads in flight together
  for (; i + 3 * stride < n; i += 4 * stride) {
    float x[4][N], w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
#pragma unroll
      for (int d = 0; d < N; ++d) x[k][d] = in.c[d][i + k * stride];
      w[k] = in.w[i + k * stride];
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) take(x[k], w[k]);
  }
  for (; i < n; i += stride) {
    float x[N];
#pragma unroll
    for (int d = 0; d < N; ++d) x[d] = in.c[d][i];
    take(x, in.w[i]);
  }
  // warp, then block reduction: one set of atomics per CTA (same-address atomics from every
  // warp of a large grid serialise at the L2)
  __shared__ uint32_t s_red[8][2 * N + 2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int d = 0; d < N; ++d) {
    emn[d] = warp_min_u(emn[d]);
    emx[d] = warp_max_u(emx[d]);
  }
  wmax = warp_max_u(wmax);
  const bool wbad = __any_sync(0xffffffffu, bad);
  if (lane == 0) {
#pragma unroll
    for (int d = 0; d < N; ++d) {
      s_red[warp][d] = emn[d];
      s_red[warp][N + d] = emx[d];
    }
    s_red[warp][2 * N] = wmax;
    s_red[warp][2 * N + 1] = wbad ? 1u : 0u;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const int nw = blockDim.x >> 5;
    for (int w = 1; w < nw; ++w) {
#pragma unroll
      for (int d = 0; d < N; ++d) {
        s_red[0][d] = min(s_red[0][d], s_red[w][d]);
        s_red[0][N + d] = max(s_red[0][N + d], s_red[w][N + d]);
      }
      s_red[0][2 * N] = max(s_red[0][2 * N], s_red[w][2 * N]);
      s_red[0][2 * N + 1] |= s_red[w][2 * N + 1];
    }
#pragma unroll
    for (int d = 0; d < N; ++d) {
      atomicMin(&g->enc_min[d], s_red[0][d]);
      atomicMax(&g->enc_max[d], s_red[0][N + d]);
    }
    atomicMax(&g->wmax_bits, s_red[0][2 * N]);
    if (s_red[0][2 * N + 1]) atomicOr(&st->nonfinite, 1u);
  }
}

// Event of point i.  Events are contiguous, ascending point ranges: chunk_ev holds the event of
// the first point of i's 1024-point chunk, and the events that start later inside the chunk are
// stepped over (a few steps at most for events of 100 points and more), which replaces a binary
// search of about log2(E) dependent loads.  Without the table (one event, or a workspace
// without it) the binary search.
__device__ __forceinline__ int event_of(const int32_t* __restrict__ ev_pt, const int32_t* __restrict__ chunk_ev,
                                        int E, int i) {
  if (E == 1) return 0;
  if (!chunk_ev) return find_event(ev_pt, E, i);
  int e = __ldg(chunk_ev + (i >> kEvChunkShift));
  while (__ldg(ev_pt + e + 1) <= i) ++e;
  return e;
}

// Event of point i, looked up once per warp when the warp's points share one event (the usual
// case: events are contiguous ranges of points) and per lane otherwise.
__device__ __forceinline__ int warp_event(const int32_t* __restrict__ ev_pt, const int32_t* __restrict__ chunk_ev,
                                          int E, int i, bool active, bool& uniform) {
  const unsigned am = __activemask();
  const int first = __shfl_sync(am, i, __ffs(am) - 1);
  const int last = __shfl_sync(am, i, 31 - __clz(am));
  const int e0 = event_of(ev_pt, chunk_ev, E, first);
  uniform = last < ev_pt[e0 + 1];
  return uniform ? e0 : (active ? event_of(ev_pt, chunk_ev, E, i) : e0);
}

// The chunk table of event_of: chunk c (points [1024 c, 1024 c + 1024)) gets the event that
// holds its first point; every non-empty event writes the chunks whose first point it holds.
__global__ void __launch_bounds__(256) k_event_chunks(int E, const int32_t* __restrict__ ev_pt,
                                                      int32_t* __restrict__ chunk_ev) {
  const int stride = gridDim.x * blockDim.x;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < E; e += stride) {
    const int a = ev_pt[e], b = ev_pt[e + 1];
    if (a >= b) continue;
    for (int c = (a + (1 << kEvChunkShift) - 1) >> kEvChunkShift; c <= (b - 1) >> kEvChunkShift; ++c) chunk_ev[c] = e;
  }
}

// Bounding box and largest |weight| of many events.  Every warp takes spans of `span`
// consecutive points (a multiple of 32) and keeps a running box while its 32-point groups stay
// inside one event, so a span inside an event costs one warp reduction and 2N + 1 atomics; a
// group that straddles events falls back to per-lane atomics.
template <int N>
__global__ void __launch_bounds__(256) k_bbox_events(InPtrs in, int n, int E, const int32_t* __restrict__ ev_pt,
                                                     const int32_t* __restrict__ chunk_ev, EvGrid* eg, DevStatus* st,
                                                     int span) {
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  bool bad = false;
  for (int base = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * span; base < n; base += nwarps * span) {
    const int end = min(n, base + span);
    {
      // the usual case, a span inside one event: four 32-point groups per step with their loads
      // in flight together, one warp reduction and 2N + 1 atomics
      const int e0 = event_of(ev_pt, chunk_ev, E, base);
      if (ev_pt[e0 + 1] >= end) {
        uint32_t bmn[N], bmx[N], bw = 0;
#pragma unroll
        for (int d = 0; d < N; ++d) {
          bmn[d] = 0xffffffffu;
          bmx[d] = 0;
        }
        for (int i0 = base; i0 < end; i0 += 128) {
          float xs[4][N], wv[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int i = min(i0 + 32 * k + lane, end - 1);  // lanes past the end repeat the last point
#pragma unroll
            for (int d = 0; d < N; ++d) xs[k][d] = in.c[d][i];
            wv[k] = in.w[i];
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) {
#pragma unroll
            for (int d = 0; d < N; ++d) {
              bad |= !isfinite(xs[k][d]);
              const uint32_t u = enc_float(xs[k][d]);
              bmn[d] = min(bmn[d], u);
              bmx[d] = max(bmx[d], u);
            }
            bad |= !isfinite(wv[k]);
            bw = max(bw, __float_as_uint(fabsf(wv[k])));
          }
        }
#pragma unroll
        for (int d = 0; d < N; ++d) {
          bmn[d] = warp_min_u(bmn[d]);
          bmx[d] = warp_max_u(bmx[d]);
        }
        bw = warp_max_u(bw);
        if (lane == 0) {
#pragma unroll
          for (int d = 0; d < N; ++d) {
            atomicMin(&eg[e0].enc_min[d], bmn[d]);
            atomicMax(&eg[e0].enc_max[d], bmx[d]);
          }
          atomicMax(&eg[e0].wmax_bits, bw);
        }
        continue;
      }
    }
    int cur = -1;  // event of the running box (warp-uniform), -1: none
    uint32_t amn[N], amx[N], aw = 0;
#pragma unroll
    for (int d = 0; d < N; ++d) amn[d] = amx[d] = 0;
    auto flush = [&]() {
#pragma unroll
      for (int d = 0; d < N; ++d) {
        amn[d] = warp_min_u(amn[d]);
        amx[d] = warp_max_u(amx[d]);
      }
      aw = warp_max_u(aw);
      if (lane == 0) {
#pragma unroll
        for (int d = 0; d < N; ++d) {
          atomicMin(&eg[cur].enc_min[d], amn[d]);
          atomicMax(&eg[cur].enc_max[d], amx[d]);
        }
        atomicMax(&eg[cur].wmax_bits, aw);
      }
    };
    for (int i0 = base; i0 < end; i0 += 32) {
      const int i = min(i0 + lane, end - 1);  // lanes past the end repeat the last point
      bool uniform;
      const int e = warp_event(ev_pt, chunk_ev, E, i, true, uniform);
      uint32_t emn[N];
#pragma unroll
      for (int d = 0; d < N; ++d) {
        const float x = in.c[d][i];
        bad |= !isfinite(x);
        emn[d] = enc_float(x);
      }
      const float w = in.w[i];
      bad |= !isfinite(w);
      const uint32_t wm = __float_as_uint(fabsf(w));
      if (uniform && e == cur) {
#pragma unroll
        for (int d = 0; d < N; ++d) {
          amn[d] = min(amn[d], emn[d]);
          amx[d] = max(amx[d], emn[d]);
        }
        aw = max(aw, wm);
        continue;
      }
      if (cur >= 0) flush();
      if (uniform) {
        cur = e;
#pragma unroll
        for (int d = 0; d < N; ++d) amn[d] = amx[d] = emn[d];
        aw = wm;
      } else {
        cur = -1;
#pragma unroll
        for (int d = 0; d < N; ++d) {
          atomicMin(&eg[e].enc_min[d], emn[d]);
          atomicMax(&eg[e].enc_max[d], emn[d]);
        }
        atomicMax(&eg[e].wmax_bits, wm);
      }
    }
    if (cur >= 0) flush();
  }
  if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(&st->nonfinite, 1u);
}

// Tile size (max - min) / nperdim in FP32 (ComputeTiles.hpp:20-23), per event.
template <int N>
__global__ void k_grid(int E, EvGrid* eg) {
  const int stride = gridDim.x * blockDim.x;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < E; e += stride) {
    EvGrid& g = eg[e];
#pragma unroll
    for (int d = 0; d < N; ++d) {
      const float mn = dec_float(g.enc_min[d]);
      const float mx = dec_float(g.enc_max[d]);
      g.mn[d] = mn;
      g.mx[d] = mx;
      g.size[d] = fdiv(fsub(mx, mn), (float)g.nperdim);
    }
  }
}

// Event-major global tile key of every point (TilesView.hpp:53-61, exact integers).
template <int N>
__global__ void __launch_bounds__(256) k_bin(const KParams kp, InPtrs in, Events ev,
                                             uint32_t* __restrict__ keys) {
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kp.n; i += stride) {
    bool uniform;
    const EvGrid* g = ev.eg + warp_event(ev.pt, ev.chunk_ev, kp.n_events, i, true, uniform);
    int gb = g->tile_base;
#pragma unroll
    for (int d = 0; d < N; ++d)
      gb += g->stride[d] * get_bin(in.c[d][i], g->mn[d], g->mx[d], g->size[d], kp.wrapped[d] != 0, g->nperdim);
    keys[i] = (uint32_t)gb;
  }
}

template <int N>
__global__ void __launch_bounds__(256) k_gather(InPtrs in, int n, const int32_t* __restrict__ perm,
                                                float4* __restrict__ rec_w, DevStatus* st) {
  const int stride = gridDim.x * blockDim.x;
  for (int pos = blockIdx.x * blockDim.x + threadIdx.x; pos < n; pos += stride) {
    const int i = perm[pos];
    if (dcheck_bad(st, i, n, kChkGatherPerm)) continue;
    float x[N];
#pragma unroll
    for (int d = 0; d < N; ++d) x[d] = in.c[d][i];
    store_rec<N>(rec_w, pos, x, in.w[i]);
  }
}

// Morton bits per dimension of the fine order inside a tile (16 bits per key in total, so the
// order -- and the spatial-order sums -- depend only on the tile's own points).
template <int N>
struct MortonBits {
  static constexpr int kPerDim = N == 1 ? 16 : (16 / N > 0 ? 16 / N : 1);
  static constexpr int kBits = kPerDim * N;
};

// Morton bits the tile-internal order sorts on: the top bits of the interleaved code, a fixed
// count per dimension, so an event's record order (and with it the bits of its densities) never
// depends on the batch around it or on which of the two sort paths built it.  Two dimensions keep
// 15 of 16 bits, so a (tile, Morton) composite key fits 32 bits up to 2^17 tiles.
template <int N>
struct MortonSortBits {
  static constexpr int kBits = N == 2 ? 15 : MortonBits<N>::kBits;
};

// The bits of c (below 2^kPerDim) moved to positions 0, N, 2N, ... of a Morton code.
template <int N>
__device__ __forceinline__ uint32_t spread_bits(uint32_t c) {
  if constexpr (N == 1) {
    return c;
  } else if constexpr (N == 2) {  // 8 bits
    c = (c | (c << 4)) & 0x0f0fu;
    c = (c | (c << 2)) & 0x3333u;
    return (c | (c << 1)) & 0x5555u;
  } else {
    uint32_t m = 0;
#pragma unroll
    for (int bit = 0; bit < MortonBits<N>::kPerDim; ++bit) m |= ((c >> bit) & 1u) << (bit * N);
    return m;
  }
}

// Morton key of every tile-sorted record inside its tile (tile keys are read from tile_keys).
template <int N>
__global__ void __launch_bounds__(256) k_morton_keys(const KParams kp, Events ev, const float4* __restrict__ rec,
                                                     const uint32_t* __restrict__ tile_keys,
                                                     uint32_t* __restrict__ keys) {
  constexpr int bpd = MortonBits<N>::kPerDim;
  const float scale = (float)(1u << bpd);
  const int stride = gridDim.x * blockDim.x;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < kp.n; q += stride) {
    const uint32_t t = tile_keys[q];
    bool uniform;  // tile-sorted positions are event-major: event e holds [ev.pt[e], ev.pt[e + 1])
    const EvGrid* g = ev.eg + warp_event(ev.pt, ev.chunk_ev, kp.n_events, q, true, uniform);
    int hb[N];
    home_bins<N>(g, (int)t, hb);
    float x[N], pl;
    load_rec<N>(rec, q, x, pl);
    uint32_t m = 0;
#pragma unroll
    for (int d = 0; d < N; ++d) {
      // position inside the tile from getBin's quotient, as in k_bin_composite
      const float xd = kp.wrapped[d] ? normalize_coord(x[d], g->mn[d], g->mx[d]) : x[d];
      const float qd = fdiv(fsub(xd, g->mn[d]), g->size[d]);
      int c = g->size[d] > 0.0f ? (int)((qd - (float)hb[d]) * scale) : 0;
      c = c < 0 ? 0 : (c > (1 << bpd) - 1 ? (1 << bpd) - 1 : c);
      m |= spread_bits<N>((uint32_t)c) << d;
    }
    keys[q] = m >> (MortonBits<N>::kBits - MortonSortBits<N>::kBits);
  }
}

// Tile key of every record in the Morton-sorted order (second, stable sort by tile).
__global__ void __launch_bounds__(256) k_tile_of(const uint32_t* __restrict__ tile_keys,
                                                 const int32_t* __restrict__ mq, int n, uint32_t* __restrict__ out) {
  const int stride = gridDim.x * blockDim.x;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += stride) out[p] = tile_keys[mq[p]];
}

// Composite key (tile << mbits | Morton code of the point inside its tile, top mbits bits) of
// every point, for the single sort that yields the (tile, Morton) order directly.  Every thread
// takes four points per step, their coordinates loaded together before the keys are computed.
template <int N>
__global__ void __launch_bounds__(256) k_bin_composite(const KParams kp, InPtrs in, Events ev, int mbits,
                                                       uint32_t* __restrict__ keys) {
  constexpr int bpd = MortonBits<N>::kPerDim;
  constexpr int kPer = 4;
  const float scale = (float)(1u << bpd);
  for (int base = blockIdx.x * (256 * kPer); base < kp.n; base += gridDim.x * 256 * kPer) {
    float xs[kPer][N];
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const int i = min(base + k * 256 + (int)threadIdx.x, kp.n - 1);
#pragma unroll
      for (int d = 0; d < N; ++d) xs[k][d] = in.c[d][i];
    }
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const int i = base + k * 256 + (int)threadIdx.x;
      if (i >= kp.n) break;
      bool uniform;
      const EvGrid* g = ev.eg + warp_event(ev.pt, ev.chunk_ev, kp.n_events, i, true, uniform);
      int gb = g->tile_base;
      uint32_t m = 0;
#pragma unroll
      for (int d = 0; d < N; ++d) {
        // getBin without wrapped coordinates (the composite sort is only taken without them):
        // the quotient also places the point inside its tile for the Morton code
        const float q = fdiv(fsub(xs[k][d], g->mn[d]), g->size[d]);
        int b = cvt_i32(q);
        b = b < g->nperdim - 1 ? b : g->nperdim - 1;
        b = b > 0 ? b : 0;
        gb += g->stride[d] * b;
        int c = g->size[d] > 0.0f ? (int)((q - (float)b) * scale) : 0;
        c = c < 0 ? 0 : (c > (1 << bpd) - 1 ? (1 << bpd) - 1 : c);
        m |= spread_bits<N>((uint32_t)c) << d;
      }
      keys[i] = ((uint32_t)gb << mbits) | (m >> (MortonBits<N>::kBits - mbits));
    }
  }
}

template <int N>
__global__ void __launch_bounds__(256) k_gather_morton(const float4* __restrict__ rec_r, int n,
                                                       const int32_t* __restrict__ mq, float4* __restrict__ rec_m) {
  constexpr int W = Rec<N>::kWords;
  const int stride = gridDim.x * blockDim.x;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += stride) {
    const int q = mq[p];
#pragma unroll
    for (int k = 0; k < W; ++k) rec_m[(size_t)p * W + k] = __ldg(rec_r + (size_t)q * W + k);
  }
}

// ---- stage 1 in one launch: single events of up to kBuildPoints points, small batches ----------
// A cluster of CTAs takes one event through the whole stage: bounding box, grid, tile and Morton keys,
// the stable radix sorts, records, tile offsets, chunks and the symmetric density's block boxes.
// Its CTAs exchange digit counts through distributed shared memory and the keys through L2, with a
// cluster barrier between steps.  Bound by the latency of its steps (a radix pass of 16k points takes
// about 5 us, one of 1000 points 2 us), where a launch takes 2 to 3 us: stage 1 of a flat event was
// 24 launches, 125 us of direct launches for 16k points against 40 us, 163 against 73 us for 65k.

// Shared memory of one CTA of a build cluster.
template <int N, int W>
struct BuildSmem {
  uint32_t cnt[W][kRadix];  // digit counters of every warp, then its next positions
  uint32_t tot[2][kRadix];  // digit counts of the CTA, read by the other CTAs (two passes in turn)
  uint32_t scan[33];
  uint32_t red[W][2 * N + 2];
  uint32_t box[2 * N + 2];  // the CTA's part of the bounding box
  float mn[N], size[N], mx[N];
};

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// The address of a shared-memory word of the cluster's CTA `rank`, and a load from it.
__device__ __forceinline__ uint32_t load_remote(const uint32_t* p, uint32_t rank) {
  uint32_t a = (uint32_t)__cvta_generic_to_shared(p), r, v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(r) : "memory");
  return v;
}

// Block-wide exclusive scan of one value per thread over W warps; the total goes to *tot.
template <int W>
__device__ __forceinline__ uint32_t build_scan(uint32_t* s, uint32_t v, int lane, int warp, uint32_t* tot) {
  uint32_t inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) s[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    const uint32_t x = lane < W ? s[lane] : 0u;
    uint32_t xi = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, xi, o);
      if (lane >= o) xi += t;
    }
    s[lane] = xi - x;
    if (lane == 31) s[32] = xi;
  }
  __syncthreads();
  const uint32_t r = s[warp] + inc - v;
  *tot = s[32];
  __syncthreads();
  return r;
}

// One stable radix pass over the event's n (key, value) pairs by the digit at `shift`; a null vin
// stands for the points pt..pt+n-1.  Warp w of the cluster takes the pairs [w L, w L + L) in order.
template <int N, int W>
__device__ void build_pass(BuildSmem<N, W>& sm, int pass, const uint32_t* kin, const int32_t* vin, uint32_t* kout,
                           int32_t* vout, int n, int pt, int shift, uint32_t rank, uint32_t ranks, int lane, int warp) {
  constexpr int K = 4;  // loads in flight per lane
  const int L = ((n + (int)ranks * W - 1) / ((int)ranks * W) + 31) & ~31;
  const int b = min(n, ((int)rank * W + warp) * L), e = min(n, b + L);
  uint32_t* cnt = sm.cnt[warp];
  for (int d = lane; d < kRadix; d += 32) cnt[d] = 0u;
  __syncwarp();
  for (int i0 = b + lane; i0 < e; i0 += 32 * K) {
    uint32_t k[K];
#pragma unroll
    for (int j = 0; j < K; ++j) k[j] = i0 + 32 * j < e ? __ldcg(kin + i0 + 32 * j) : 0u;
#pragma unroll
    for (int j = 0; j < K; ++j)
      if (i0 + 32 * j < e) atomicAdd(&cnt[(k[j] >> shift) & (kRadix - 1)], 1u);
  }
  __syncthreads();
  const int t = threadIdx.x;
  uint32_t* tot = sm.tot[pass & 1];
  if (t < kRadix) {
    uint32_t run = 0;
#pragma unroll 8
    for (int w = 0; w < W; ++w) {
      const uint32_t c = sm.cnt[w][t];
      sm.cnt[w][t] = run;
      run += c;
    }
    tot[t] = run;
  }
  cluster_barrier();
  uint32_t before = 0, all = 0;
  if (t < kRadix) {
    for (uint32_t r = 0; r < ranks; ++r) {
      const uint32_t v = load_remote(tot + t, r);
      before += r < rank ? v : 0u;
      all += v;
    }
  }
  uint32_t sum;
  const uint32_t base = build_scan<W>(sm.scan, t < kRadix ? all : 0u, lane, warp, &sum) + before;
  if (t < kRadix) {
#pragma unroll 8
    for (int w = 0; w < W; ++w) sm.cnt[w][t] += base;
  }
  __syncthreads();
  const uint32_t lt = (1u << lane) - 1u;
  for (int i0 = b; i0 < e; i0 += 32 * K) {
    uint32_t k[K];
    int32_t v[K];
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const int i = i0 + 32 * j + lane;
      k[j] = i < e ? __ldcg(kin + i) : 0u;
      v[j] = i < e ? (vin ? __ldcg(vin + i) : pt + i) : 0;
    }
#pragma unroll
    for (int j = 0; j < K; ++j) {
      if (i0 + 32 * j >= e) break;
      const bool valid = i0 + 32 * j + lane < e;
      const uint32_t d = (k[j] >> shift) & (kRadix - 1);
      uint32_t peers = __ballot_sync(0xffffffffu, valid);
      peers = valid ? peers : ~peers;
#pragma unroll
      for (int bit = 0; bit < kRadixBits; ++bit) {
        const bool one = (d >> bit) & 1u;
        const uint32_t bb = __ballot_sync(0xffffffffu, one);
        peers &= one ? bb : ~bb;
      }
      const uint32_t place = valid ? cnt[d] + (uint32_t)__popc(peers & lt) : 0u;
      __syncwarp();
      if (valid) {
        if ((peers & lt) == 0) cnt[d] += (uint32_t)__popc(peers);
        kout[place] = k[j];
        vout[place] = v[j];
      }
      __syncwarp();
    }
  }
  cluster_barrier();
}

// Records of a build cluster's arrays, written by other CTAs of the cluster in this launch.
template <int N>
__device__ __forceinline__ void load_rec_cg(const float4* rec, int pos, float* x, float& payload) {
  constexpr int WD = Rec<N>::kWords;
  float buf[4 * WD];
#pragma unroll
  for (int k = 0; k < WD; ++k) {
    const float4 v = __ldcg(rec + (size_t)pos * WD + k);
    buf[4 * k] = v.x, buf[4 * k + 1] = v.y, buf[4 * k + 2] = v.z, buf[4 * k + 3] = v.w;
  }
#pragma unroll
  for (int d = 0; d < N; ++d) x[d] = buf[d];
  payload = buf[Rec<N>::kPayload];
}

// The buffers of k_build; `two` sorts give the tile order by index and the Morton order, one the
// (tile, Morton) order alone (the symmetric density's).
struct BuildBufs {
  uint32_t *k0, *k1, *k2;   // keys: composite keys, the other buffer of their sort, first pass of the tile sort
  int32_t *va, *vb;         // values of the composite sort, pass by pass
  int32_t *perm, *vt;       // result of the tile sort, its first pass
  int32_t* inv;             // tile-sorted position of every point
  float4* rec_w;
  int32_t* off;
  uint32_t *chunk_off, *tblk_off;
  int32_t* chunk_tile;
  uint32_t* chunk_total;
  float4* tblk;
  int64_t* rho_fix;
  uint32_t* seed_bits;
  int32_t *ev_pt, *ev_tile, *ev_chunk;
  DevStatus* st;
};

// Event e by one cluster of `ranks` CTAs.
template <int N, int W>
__device__ __forceinline__ void build_event(BuildSmem<N, W>& sm, const KParams& kp, const InPtrs& in, EvGrid* eg,
                                            const BuildBufs& o, bool two, int mbits, int tile_passes, int passes, int e,
                                            uint32_t rank, uint32_t ranks) {
  const int lane = lane_id(), warp = threadIdx.x >> 5;
  EvGrid* g = eg + e;
  const bool single = kp.n_events == 1;
  const int n = single ? kp.n : g->pt_count, pt = single ? 0 : g->pt_base;
  const int ntiles = single ? kp.ntiles : g->ntiles, tile_base = single ? 0 : g->tile_base;
  const int npd = single ? kp.nperdim0 : g->nperdim;
  const int tid = rank * (32 * W) + threadIdx.x, step = ranks * (32 * W);
  // the call's state (k_init's work; a batch runs k_init before)
  if (single) {
    if (rank == 0)
      for (int k = threadIdx.x; k < (int)(sizeof(DevStatus) / 4); k += 32 * W) reinterpret_cast<uint32_t*>(o.st)[k] = 0u;
    for (int k = tid; k < (n + 31) / 32; k += step) o.seed_bits[k] = 0u;
    if (tid == 0) {
      g->nperdim = npd;
      g->ntiles = ntiles;
      g->tile_base = 0;
      g->pt_base = 0;
      g->pt_count = n;
      for (int d = 0; d < kMaxDim; ++d) g->stride[d] = kp.stride0[d];
      o.ev_pt[0] = 0;
      o.ev_pt[1] = n;
      o.ev_tile[0] = 0;
      o.ev_tile[1] = ntiles;
    }
  } else if (o.ev_chunk) {
    for (int c = ((pt + (1 << kEvChunkShift) - 1) >> kEvChunkShift) + tid; c <= (pt + n - 1) >> kEvChunkShift; c += step)
      o.ev_chunk[c] = e;
  }
  if (o.rho_fix)
    for (int k = tid; k < n; k += step) o.rho_fix[pt + k] = 0;
  // bounding box, largest |weight|, finite values
  {
    uint32_t emn[N], emx[N], wmax = 0u;
    bool bad = false;
#pragma unroll
    for (int d = 0; d < N; ++d) {
      emn[d] = 0xffffffffu;
      emx[d] = 0u;
    }
#pragma unroll 2
    for (int i = tid; i < n; i += step) {
#pragma unroll
      for (int d = 0; d < N; ++d) {
        const float x = in.c[d][pt + i];
        bad |= !isfinite(x);
        const uint32_t u = enc_float(x);
        emn[d] = min(emn[d], u);
        emx[d] = max(emx[d], u);
      }
      const float w = in.w[pt + i];
      bad |= !isfinite(w);
      wmax = max(wmax, __float_as_uint(fabsf(w)));
    }
#pragma unroll
    for (int d = 0; d < N; ++d) {
      const uint32_t a = warp_min_u(emn[d]), z = warp_max_u(emx[d]);
      if (lane == 0) {
        sm.red[warp][d] = ~a;  // every entry is combined by maximum
        sm.red[warp][N + d] = z;
      }
    }
    wmax = warp_max_u(wmax);
    bad = __any_sync(0xffffffffu, bad);
    if (lane == 0) {
      sm.red[warp][2 * N] = wmax;
      sm.red[warp][2 * N + 1] = bad ? 1u : 0u;
    }
    __syncthreads();
    if (threadIdx.x < 2 * N + 2) {
      uint32_t v = 0u;
      for (int w = 0; w < W; ++w) v = max(v, sm.red[w][threadIdx.x]);
      sm.box[threadIdx.x] = v;
    }
    cluster_barrier();
    if (threadIdx.x < 2 * N + 2) {
      uint32_t v = 0u;
      for (uint32_t r = 0; r < ranks; ++r) v = max(v, load_remote(sm.box + threadIdx.x, r));
      sm.red[0][threadIdx.x] = v;
    }
    __syncthreads();
    if (threadIdx.x < N) {
      const int d = threadIdx.x;
      // tile size (max - min) / nperdim in FP32 (ComputeTiles.hpp:20-23)
      const float mn = dec_float(~sm.red[0][d]), mx = dec_float(sm.red[0][N + d]);
      const float size = fdiv(fsub(mx, mn), (float)npd);
      sm.mn[d] = mn;
      sm.mx[d] = mx;
      sm.size[d] = size;
      if (rank == 0) {
        g->mn[d] = mn;
        g->mx[d] = mx;
        g->size[d] = size;
      }
    }
    if (rank == 0 && threadIdx.x == 32) {
      g->seed_candidates = 0;
      g->wmax_bits = sm.red[0][2 * N];
      if (sm.red[0][2 * N + 1]) atomicOr(&o.st->nonfinite, 1u);
    }
    __syncthreads();
  }
  // composite keys: tile of the event's grid, then the Morton code inside the tile
  {
    constexpr int bpd = MortonBits<N>::kPerDim;
    const float scale = (float)(1u << bpd);
    for (int i = tid; i < n; i += step) {
      int gb = 0;
      uint32_t m = 0;
#pragma unroll
      for (int d = 0; d < N; ++d) {
        float x = in.c[d][pt + i];
        if (kp.wrapped[d]) x = normalize_coord(x, sm.mn[d], sm.mx[d]);
        const float q = fdiv(fsub(x, sm.mn[d]), sm.size[d]);
        int b = cvt_i32(q);
        b = b < npd - 1 ? b : npd - 1;
        b = b > 0 ? b : 0;
        gb = gb * npd + b;
        int c = sm.size[d] > 0.0f ? (int)((q - (float)b) * scale) : 0;
        c = c < 0 ? 0 : (c > (1 << bpd) - 1 ? (1 << bpd) - 1 : c);
        m |= spread_bits<N>((uint32_t)c) << d;
      }
      o.k0[pt + i] = ((uint32_t)gb << mbits) | (m >> (MortonBits<N>::kBits - mbits));
    }
  }
  cluster_barrier();
  int pass = 0;
  if (two) {
    for (int p = 0; p < tile_passes; ++p, ++pass) {
      const bool last = p + 1 == tile_passes;
      build_pass<N, W>(sm, pass, p == 0 ? o.k0 + pt : o.k2 + pt, p == 0 ? nullptr : o.vt + pt, last ? o.k1 + pt : o.k2 + pt,
                       last ? o.perm + pt : o.vt + pt, n, pt, mbits + 8 * p, rank, ranks, lane, warp);
    }
  }
  for (int p = 0; p < passes; ++p, ++pass)
    build_pass<N, W>(sm, pass, (p & 1 ? o.k1 : o.k0) + pt, p == 0 ? nullptr : (p & 1 ? o.va : o.vb) + pt,
                     (p & 1 ? o.k0 : o.k1) + pt, (p & 1 ? o.vb : o.va) + pt, n, pt, 8 * p, rank, ranks, lane, warp);
  const uint32_t* sorted = (passes & 1 ? o.k1 : o.k0) + pt;
  const int32_t* by_morton = (passes & 1 ? o.va : o.vb) + pt;
  int32_t* mq = (passes & 1 ? o.vb : o.va) + pt;
  // records, tile offsets
  for (int base = tid & ~31; base <= n; base += step) {
    const int q = base + lane;
    int prev = 0, cur = -1;  // tiles that start at q: prev + 1 .. cur
    if (q <= n) {
      prev = q > 0 ? (int)(__ldcg(sorted + q - 1) >> mbits) : -1;
      cur = q < n ? (int)(__ldcg(sorted + q) >> mbits) : ntiles;
    }
    const bool far = cur - prev > 32;
    if (!far)
      for (int t = prev + 1; t <= cur; ++t) o.off[tile_base + t] = pt + q;
    for (unsigned m = __ballot_sync(0xffffffffu, far); m; m &= m - 1) {
      const int src = __ffs(m) - 1;
      const int p = __shfl_sync(0xffffffffu, prev, src), c = __shfl_sync(0xffffffffu, cur, src);
      for (int t = p + 1 + lane; t <= c; t += 32) o.off[tile_base + t] = pt + base + src;
    }
    if (q < n) {
      const int i = __ldcg(two ? o.perm + pt + q : by_morton + q);
      if (!dcheck_bad(o.st, i, kp.n, kChkGatherPerm)) {
        float x[N];
#pragma unroll
        for (int d = 0; d < N; ++d) x[d] = in.c[d][i];
        store_rec<N>(o.rec_w, pt + q, x, in.w[i]);
        if (two) o.inv[i] = pt + q;
      }
    }
  }
  cluster_barrier();
  if (two)
    for (int p = tid; p < n; p += step) {
      const int i = __ldcg(by_morton + p);
      if (!dcheck_bad(o.st, i, kp.n, kChkGatherPerm)) mq[p] = __ldcg(o.inv + i);
    }
  // chunks of kChunk home points and blocks of 32 points of every tile; an event of a batch has the
  // slots that its points and tiles can need at most, the unused ones are marked
  const int slot0 = single ? 0 : pt / kChunk + tile_base, blk0 = single ? 0 : pt / 32 + tile_base;
  if (rank == 0) {
    uint32_t chunks = 0, blocks = 0;
    for (int t0 = 0; t0 < ntiles; t0 += 32 * W) {
      const int t = t0 + (int)threadIdx.x;
      const int cnt = t < ntiles ? __ldcg(o.off + tile_base + t + 1) - __ldcg(o.off + tile_base + t) : 0;
      const uint32_t nch = (uint32_t)((cnt + kChunk - 1) / kChunk), nbl = (uint32_t)((cnt + 31) / 32);
      uint32_t sum;
      const uint32_t ce = chunks + build_scan<W>(sm.scan, nch, lane, warp, &sum);
      chunks += sum;
      const uint32_t be = blocks + build_scan<W>(sm.scan, nbl, lane, warp, &sum);
      blocks += sum;
      if (t < ntiles) {
        o.chunk_off[tile_base + t] = (uint32_t)slot0 + ce;
        if (o.tblk_off) o.tblk_off[tile_base + t] = (uint32_t)blk0 + be;
        for (uint32_t c = 0; c < nch; ++c) o.chunk_tile[slot0 + ce + c] = tile_base + t;
      }
    }
    if (single) {
      if (threadIdx.x == 0) *o.chunk_total = chunks;
    } else {
      const int end = e + 1 < kp.n_events ? (pt + n) / kChunk + tile_base + ntiles : kp.n / kChunk + kp.ntiles + 1;
      for (int c = slot0 + (int)chunks + (int)threadIdx.x; c < end; c += 32 * W) o.chunk_tile[c] = -1;
    }
    if (threadIdx.x == 0) sm.scan[0] = chunks;
  }
  if (!o.tblk) return;  // (no CTA reads another's shared memory any more)
  cluster_barrier();
  const int nblocks = kChunkWarps * (int)load_remote(sm.scan, 0);
  for (int sl = rank * W + warp; sl < nblocks; sl += ranks * W) {
    const int t = __ldcg(o.chunk_tile + slot0 + sl / kChunkWarps);
    const int b = (slot0 + sl / kChunkWarps - (int)__ldcg(o.chunk_off + t)) * kChunkWarps + sl % kChunkWarps;
    const int first = __ldcg(o.off + t) + (b << 5);
    const int cnt = min(32, __ldcg(o.off + t + 1) - first);
    if (cnt <= 0) continue;
    float x[N], w;
    load_rec_cg<N>(o.rec_w, first + min(lane, cnt - 1), x, w);
    write_block_box<N>(o.tblk, (int)__ldcg(o.tblk_off + t) + b, x, w);
  }
  cluster_barrier();  // sm.scan[0] of the first CTA is read by all
}

// An event per cluster.  The clusters of a launch share its events by the sizes that the hardware
// reports, whatever was asked for (an executable graph updated in place has kept an older launch's).
template <int N, int W>
__global__ void __launch_bounds__(32 * W) k_build(const KParams kp, InPtrs in, EvGrid* eg, BuildBufs o, bool two,
                                                  int mbits, int tile_passes, int passes) {
  __shared__ BuildSmem<N, W> sm;
  uint32_t rank, ranks;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(ranks));
  const int clusters = gridDim.x / ranks;
  for (int e = blockIdx.x / ranks; e < kp.n_events; e += clusters) {
    build_event<N, W>(sm, kp, in, eg, o, two, mbits, tile_passes, passes, e, rank, ranks);
    if (e + clusters < kp.n_events) cluster_barrier();  // the next event takes the same shared memory
  }
}

// ---- chunks ---------------------------------------------------------------------
// Home points of every tile are taken in the tile's fine Morton order (so 32 consecutive points are
// close together at the data's own density scale), cut into chunks of kChunk points; one CTA
// processes one chunk, so a heavy tile is spread over many CTAs.

// Chunks of kChunk and blocks of 32 points of every tile.
__global__ void k_tile_counts(int ntiles, const int32_t* __restrict__ off, uint32_t* __restrict__ chunk_count,
                              uint32_t* __restrict__ blk_count) {
  const int stride = gridDim.x * blockDim.x;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < ntiles; t += stride) {
    const int cnt = off[t + 1] - off[t];
    chunk_count[t] = (uint32_t)((cnt + kChunk - 1) / kChunk);
    if (blk_count) blk_count[t] = (uint32_t)((cnt + 31) / 32);
  }
}

__global__ void k_chunk_map(int ntiles, const int32_t* __restrict__ off, const uint32_t* __restrict__ chunk_off,
                            int32_t* __restrict__ chunk_tile) {
  const int stride = gridDim.x * blockDim.x;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < ntiles; t += stride) {
    const int nch = (off[t + 1] - off[t] + kChunk - 1) / kChunk;
    const uint32_t c0 = chunk_off[t];
    for (int c = 0; c < nch; ++c) chunk_tile[c0 + c] = t;
  }
}

// Chunk of the CTA: tile, event grid and home position of this thread.
struct ChunkHome {
  int t;
  const EvGrid* g;
  int p;  // the thread's slot of the tile's home order (the chunk's first slot when not valid)
  bool valid;
};

__device__ __forceinline__ bool chunk_home(const KParams& kp, Events ev, const int32_t* __restrict__ off,
                                           const int32_t* __restrict__ chunk_tile,
                                           const uint32_t* __restrict__ chunk_off,
                                           const uint32_t* __restrict__ chunk_total, ChunkHome& h) {
  const int w = blockIdx.x;
  if (w >= (int)*chunk_total) return false;
  h.t = chunk_tile[w];
  if (h.t < 0) return false;  // a slot that its event does not need (k_build)
  const int beg = off[h.t];
  // slots are event-major: the tile's first one lies among its event's points
  h.g = ev.eg + event_of(ev.pt, ev.chunk_ev, kp.n_events, beg);
  const int start = (w - (int)chunk_off[h.t]) * kChunk;
  const int cnt = min(kChunk, off[h.t + 1] - beg - start);
  h.valid = (int)threadIdx.x < cnt;
  h.p = beg + start + (h.valid ? (int)threadIdx.x : 0);
  return true;
}

// ---- stage 2: local density --------------------------------------------------
// rho_i accumulates, in the reference's candidate order (search-box tiles
// lexicographically, ascending index inside a tile), term = k(d, i, j) * w_j for every
// candidate with d <= dc; candidates beyond dc contribute +-0 and are skipped.
//
// The homes of a warp are 32 neighbours of a tile's Morton order, so most candidates of its
// search-box tiles are out of every lane's reach: the lanes read 64 candidates at a time (in index
// order), keep those within dc of the box of the warp's homes, and append them to the warp's buffer
// in shared memory, coordinates and terms by dimension.  What is kept is summed 32 at a time, four
// candidates per load with paired differences and squares: 7 instructions a candidate, where staging
// whole tiles by bulk copy and testing every candidate took about 12.  Bound by instruction issue on
// large inputs and by the sums' own chain of additions where a scheduler has one warp: 0.66 -> 0.31 ms
// on 1M 2-D points, 67 -> 36 us on 16k (homes in Morton order as they are; grouping them by the
// tiles their search boxes reach, in a pass of 25 us, is not needed any more).
template <int N, int MT>
__global__ void __launch_bounds__(kTileThreads, (N <= 4 ? 8 : 4)) k_density(
    const KParams kp, Events ev, const int32_t* __restrict__ off, const int32_t* __restrict__ chunk_tile,
    const uint32_t* __restrict__ chunk_off, const uint32_t* __restrict__ chunk_total,
    const float4* __restrict__ rec_w, const int32_t* __restrict__ mq, float4* __restrict__ rec_r) {
  using M = Metric<N, MT>;
  // coordinates and flat-kernel terms (or weights) of the kept candidates, a ring of 128
  __shared__ ulonglong2 s_buf[kChunkWarps][N + 1][32];
  ChunkHome h;
  if (!chunk_home(kp, ev, off, chunk_tile, chunk_off, chunk_total, h)) return;
  const bool valid = h.valid;
  if (!__any_sync(0xffffffffu, valid)) return;
  const int lane = lane_id(), warp = threadIdx.x >> 5;
  const int pos = order_at(mq, h.p);
  float x[N], wi;
  load_rec<N>(rec_w, pos, x, wi);
  int hb[N], lo[N], hi[N], wl[N], wh[N];
  home_bins<N>(h.g, h.t, hb);
  lane_box<N>(kp, h.g, x, kp.dc, hb, lo, hi);
  float hlo[N], hhi[N];  // box of the warp's homes
#pragma unroll
  for (int d = 0; d < N; ++d) {
    wl[d] = warp_min_i(valid ? lo[d] : INT_MAX);
    wh[d] = warp_max_i(valid ? hi[d] : INT_MIN);
    hlo[d] = warp_min_f(valid ? x[d] : INFINITY);
    hhi[d] = warp_max_f(valid ? x[d] : -INFINITY);
  }
  const bool flat = kp.kernel_type == CLUE_KERNEL_FLAT;
  const float kflat = kp.kpar[0];
  const float tdc = kp.t_dc;
  const unsigned lt = (1u << lane) - 1u;
  unsigned long long x2[N];
#pragma unroll
  for (int d = 0; d < N; ++d) x2[d] = pk2(make_float2(x[d], x[d]));
  const unsigned long long one = pk2(make_float2(kp.one, kp.one));
  float rho = 0.0f;
  box_tiles<N>(h.g, off, hb, wl, wh, -1, lane, [&](const int* v, int, int pb, int pe) {
    bool inbox = valid;
#pragma unroll
    for (int d = 0; d < N; ++d) inbox = inbox && v[d] >= lo[d] && v[d] <= hi[d];
    if (!__any_sync(0xffffffffu, inbox)) return;
    const float thr = inbox ? tdc : -INFINITY;
    int fill = 0;        // candidates appended so far
    int self = INT_MIN;  // the home point's own number among them
    // Sums candidates [f0, f1) of the buffer (f0 a multiple of 32, at most 32 of them).
    auto sum = [&](int f0, int f1) {
      // groups of four that hold some home's own point, whose term is its weight
      const unsigned own = __reduce_or_sync(0xffffffffu, self >= f0 && self < f1 ? 1u << ((self - f0) >> 2) : 0u);
      const int q0 = (f0 >> 2) & 31;
      auto four = [&](int q, bool tail) {
        float2 s2[2];
        ulonglong2 c2[N];
#pragma unroll
        for (int d = 0; d < N; ++d) c2[d] = s_buf[warp][d][q0 + q];
        {
          unsigned long long ca[N], cb[N];
#pragma unroll
          for (int d = 0; d < N; ++d) ca[d] = c2[d].x, cb[d] = c2[d].y;
          s2[0] = partial_packed<N, MT>(x2, ca, kp.mpar, one);
          s2[1] = partial_packed<N, MT>(x2, cb, kp.mpar, one);
        }
        const float4 tv = reinterpret_cast<const float4&>(s_buf[warp][N][q0 + q]);
        float s[4] = {s2[0].x, s2[0].y, s2[1].x, s2[1].y}, tt[4] = {tv.x, tv.y, tv.z, tv.w};
        if (tail) {  // the last group's empty places
#pragma unroll
          for (int e = 1; e < 4; ++e)
            if (f0 + 4 * q + e >= f1) s[e] = INFINITY;
        }
        const bool any_own = (own >> q) & 1u;
        if (flat) {
          if (any_own) {
#pragma unroll
            for (int e = 0; e < 4; ++e) tt[e] = f0 + 4 * q + e == self ? wi : tt[e];
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) rho = s[e] <= thr ? fadd(rho, tt[e]) : rho;
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (s[e] <= thr) {
              const float kv = any_own && f0 + 4 * q + e == self
                                   ? 1.0f
                                   : kernel_value(kp.kernel_type, kp.kpar, M::finish(s[e]));
              rho = fadd(rho, fmul(kv, tt[e]));
            }
        }
      };
      if (flat && f1 - f0 == 32) {
#pragma unroll
        for (int q = 0; q < 8; ++q) four(q, false);
      } else {
        for (int q = 0; f0 + 4 * q < f1; ++q) four(q, f0 + 4 * q + 4 > f1);
      }
    };
    int done = 0;  // candidates summed so far, a multiple of 32
    float c[2][N], w[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) load_rec<N>(rec_w, min(pb + 32 * k + lane, pe - 1), c[k], w[k]);
    for (int base = pb; base < pe; base += 64) {
      const bool last = base + 64 >= pe;
      bool keep[2];
#pragma unroll
      for (int k = 0; k < 2; ++k)
        keep[k] = base + 32 * k + lane < pe && (!kp.lb_ok || lower_point<N, M>(c[k], hlo, hhi, kp.mpar) <= tdc);
      const unsigned m0 = __ballot_sync(0xffffffffu, keep[0]), m1 = __ballot_sync(0xffffffffu, keep[1]);
      const int mid = fill + __popc(m0);
#pragma unroll
      for (int k = 0; k < 2; ++k)
        if (keep[k]) {
          const int slot = ((k ? mid : fill) + __popc((k ? m1 : m0) & lt)) & 127;
#pragma unroll
          for (int d = 0; d < N; ++d) reinterpret_cast<float*>(s_buf[warp][d])[slot] = c[k][d];
          reinterpret_cast<float*>(s_buf[warp][N])[slot] = flat ? fmul(kflat, w[k]) : w[k];
        }
      const int o = pos - base;  // (a home always lies within its warp's box)
      if (o >= 0 && o < 64) self = (o < 32 ? fill : mid) + __popc((o < 32 ? m0 : m1) & ((1u << (o & 31)) - 1u));
      fill = mid + __popc(m1);
      if (!last) {  // the next ones, while the kept ones are summed
#pragma unroll
        for (int k = 0; k < 2; ++k) load_rec<N>(rec_w, min(base + 64 + 32 * k + lane, pe - 1), c[k], w[k]);
      }
      __syncwarp();
      for (; done + 32 <= fill; done += 32) sum(done, done + 32);
      if (last && done < fill) sum(done, fill);
      __syncwarp();
    }
  });
  if (valid) store_rec<N>(rec_r, pos, x, rho);
}

// ---- stage 3: nearest higher -------------------------------------------------
// j is higher than i iff rho_j > rho_i or (rho_j == rho_i, rho_j > 0, j > i) with original
// indices.  The reference keeps the first candidate of its iteration order (search-box tiles
// lexicographically, ascending index inside a tile) with the strictly smallest distance <= dm,
// i.e. the minimum of (distance, iteration rank); that minimum does not depend on the order in
// which candidates are visited, so the search here is spatial: every tile's records are also
// kept in Morton order of a fine grid inside the tile, the own tile is searched first, and a
// 32-record block is skipped when its bounding box is farther than every lane's current best
// (or than dm) or holds no density reaching the lane's.  TIE == CLUE_TIE_RHO_INDEX resolves equal
// distances by higher rho, then lower index.

// The two functions below are for equal distances: points on a lattice, or of one place.  Calls and not
// inlined, which keeps them out of the usual path's registers (4096-event batch 2.07 ms, 2.11 inlined).

// Homes `nm` of a block that still need a search home by home.  Not those with nothing higher, all
// densities being equal and the indices lower, nor those whose best so far is as near as the block's
// nearest, of this tile and of a lower index than any: pos_best (else -1).  pos, rho: the lane's candidate,
// pos_home, rho_home: the lane's home.  (16k points of one place: 0.85 ms, 13 without it.)
__device__ __noinline__ unsigned tie_block(unsigned nm, int pos_best, const int32_t* perm, int pos, float rho,
                                           float rho_home, int pos_home) {
  const int orig = __ldg(perm + pos);
  const int orig_min = warp_min_i(orig), orig_max = warp_max_i(orig);
  const float rho_max = warp_max_f(rho);
  bool skip = pos_best >= 0 && orig_min >= __ldg(perm + pos_best);
  if (rho_max <= rho_home) skip = skip || orig_max <= __ldg(perm + pos_home);
  return nm & ~__ballot_sync(0xffffffffu, skip);
}

// Of one home's candidates `om` (a lane each), the least by rounded distance, then by density (RHO_INDEX),
// then by original index, which orders the points of a tile as the iteration rank does; 0 if none is
// higher.
template <int TIE>
__device__ __noinline__ unsigned tie_least(unsigned om, float dist, float rho, float rho_home, const int32_t* perm,
                                           int pos, int pos_home) {
  const int lane = threadIdx.x & 31;
  const int orig = __ldg(perm + pos), orig_home = __ldg(perm + pos_home);
  const bool higher = ((om >> lane) & 1u) && (rho > rho_home || (rho > 0.0f && orig > orig_home));
  const float dist_min = warp_min_f(higher ? dist : INFINITY);
  bool least = higher && dist == dist_min;
  if (TIE != CLUE_TIE_REFERENCE) {
    const float rho_max = warp_max_f(least ? rho : -INFINITY);
    least = least && rho == rho_max;
  }
  const int first = warp_min_i(least ? orig : INT_MAX);
  return __ballot_sync(0xffffffffu, least && orig == first);
}

// A block is visited in one of two forms.  Where few lanes need it, it is taken home by home with
// a candidate per lane: one distance per lane, one vote, and the few candidates that pass settle
// the home's update.  Otherwise it is taken candidate by candidate with a home per lane, without
// branches: every lane keeps the two smallest keys of the block, a key being the metric value's
// bits with the candidate's number in place of the lowest five.  The smallest key names the nearest
// candidate unless the two are within one step of the shortened value (or the best so far is): such
// lanes, and those whose nearest candidate has their own density, take the first form.
// (On 512 events of the calorimeter batch a warp visits 3.3 blocks that 23 lanes need on average and
// 4.4 that 2.6 lanes need.)
// Bound by instruction issue (68% active).  A form with a vote and an update branch per candidate
// pair and lane groups for the blocks few lanes need took 7000 instructions a warp, this one 3200:
// 3.92 -> 2.00 ms on the 4096-event batch, 2.20 -> 1.10 ms on 4M 3-D points, 0.366 -> 0.193 ms on
// 1M 2-D points.  split_lanes 4 / 8 / 12 / 16 gives 2.05 / 2.00 / 2.01 / 2.06 ms and 1.21 / 1.10 /
// 1.08 / 1.09 ms on the first two.
template <int N, int MT, int TIE>
__global__ void __launch_bounds__(kTileThreads, (N <= 4 ? 8 : 4) * 128 / kTileThreads) k_nearest_higher(
    const KParams kp, Events ev, const int32_t* __restrict__ off, const int32_t* __restrict__ chunk_tile,
    const uint32_t* __restrict__ chunk_off, const uint32_t* __restrict__ chunk_total,
    const float4* __restrict__ rec_m, const int32_t* __restrict__ mq, const float4* __restrict__ blk,
    const float4* __restrict__ sblk, const int32_t* __restrict__ perm, const SeedBufs sb, const clue_outputs out,
    DevStatus* st, int split_lanes) {
  using M = Metric<N, MT>;
  ChunkHome h;
  if (!chunk_home(kp, ev, off, chunk_tile, chunk_off, chunk_total, h)) return;
  const bool valid = h.valid;
  if (!__any_sync(0xffffffffu, valid)) return;
  const int lane = lane_id(), warp = threadIdx.x >> 5;
  float x[N], rho_i;
  load_rec<N>(rec_m, h.p, x, rho_i);
  int hb[N], lo[N], hi[N];
  home_bins<N>(h.g, h.t, hb);
  lane_box<N>(kp, h.g, x, kp.dm, hb, lo, hi);
  const float tdm = kp.t_dm;
  // per warp: the homes' records, and the visited block's coordinates and densities by dimension
  __shared__ float4 s_home[kChunkWarps][32 * Rec<N>::kWords];
  __shared__ ulonglong2 s_blk[kChunkWarps][N + 1][8];
  store_rec<N>(s_home[warp], lane, x, rho_i);
  __syncwarp();
  unsigned long long x2[N];
#pragma unroll
  for (int d = 0; d < N; ++d) x2[d] = pk2(make_float2(x[d], x[d]));
  const unsigned long long one = pk2(make_float2(kp.one, kp.one));
  const float slack = M::kRoot ? 1.0f + 1.0f / 524288.0f : 1.0f;  // s range of one rounded distance
  float s_best = INFINITY;  // metric value of the nearest higher so far
  // Candidates beyond bnd cannot be nearer than the best so far (nor within dm): its distance
  // would round above delta.
  float bnd = tdm;
  int nh = -1;        // Morton position of the best so far
  int rank_best = 0;  // position of its tile in the search boxes' iteration
  const int pw = warp_min_i(valid ? h.p : INT_MAX);  // the warp's homes are pw + lane
  spatial_sweep<N, M, true>(kp, h.g, off, hb, lo, hi, valid, x, blk, sblk, rho_i, h.p, [&]() { return bnd; },
                            [&](int p0, int p1, bool need, int rank) {
    const int cnt = p1 - p0;
    // candidate p0 + j becomes the lane's best
    auto take = [&](int j, float s) {
      s_best = s;
      bnd = fminf(tdm, s * slack);
      nh = p0 + j;
      rank_best = rank;
    };
    // Full test of candidate p0 + j, within bnd and not below the lane's density: equal densities
    // are decided by the original indices, distances that may round to the best one's by the
    // rank.  The order of the calls does not matter, since the best is an exact minimum.
    auto consider = [&](int j, float s, float rho_j) {
      const int p = p0 + j;
      int orig_j = -1;
      bool higher = rho_j > rho_i;
      if (!higher && rho_j > 0.0f) {
        orig_j = __ldg(perm + order_at(mq, p));
        higher = orig_j > __ldg(perm + order_at(mq, h.p));
      }
      if (!higher) return;
      bool better;
      if (s * slack < s_best) {
        better = true;  // its distance rounds strictly below the best one's
      } else {
        // the two distances may round to the same value: decide on the rounded distances,
        // then on the iteration rank (search-box position of the tile, then the original
        // index, which orders the points of one tile in the reference's iteration)
        const float dist = M::finish(s), dbest = M::finish(s_best);
        if (dist != dbest || nh < 0) {
          better = dist < dbest;
        } else if (TIE == CLUE_TIE_REFERENCE && rank != rank_best) {
          better = rank < rank_best;
        } else {
          if (orig_j < 0) orig_j = __ldg(perm + order_at(mq, p));
          const int orig_best = __ldg(perm + order_at(mq, nh));
          if (TIE == CLUE_TIE_REFERENCE) {
            better = orig_j < orig_best;
          } else {
            float xb[N], rho_best;
            load_rec<N>(rec_m, nh, xb, rho_best);
            better = rho_j > rho_best || (rho_j == rho_best && orig_j < orig_best);
          }
        }
      }
      if (better) take(j, s);
    };
    // lane j's candidate; lanes past the block hold none (no density reaches theirs)
    float c[N], r;
    load_rec<N>(rec_m, lane < cnt ? p0 + lane : p0, c, r);
    if (lane >= cnt) r = -INFINITY;
    unsigned nm = __ballot_sync(0xffffffffu, need);
    const int k = __popc(nm);
    // home by home: about 20 instructions a home against 10 a candidate in the other form
    if (kp.lb_ok && k > split_lanes) {
      __syncwarp();  // the previous block's readers are done
#pragma unroll
      for (int d = 0; d < N; ++d) reinterpret_cast<float*>(s_blk[warp][d])[lane] = c[d];
      reinterpret_cast<float*>(s_blk[warp][N])[lane] = r;
      __syncwarp();
      const int self = h.p - p0;  // the home point itself (equal density) is not a candidate
      uint32_t k1 = 0xffffffffu, k2 = 0xffffffffu;
      for (int q = 0; 4 * q < cnt; ++q) {
        ulonglong2 c2[N];
#pragma unroll
        for (int d = 0; d < N; ++d) c2[d] = s_blk[warp][d][q];
        const float4 rv = reinterpret_cast<const float4&>(s_blk[warp][N][q]);
        const float rr[4] = {rv.x, rv.y, rv.z, rv.w};
#pragma unroll
        for (int e = 0; e < 4; e += 2) {
          unsigned long long cp[N];
#pragma unroll
          for (int d = 0; d < N; ++d) cp[d] = e ? c2[d].y : c2[d].x;
          const float2 s2 = partial_packed<N, MT>(x2, cp, kp.mpar, one);
#pragma unroll
          for (int f = 0; f < 2; ++f) {
            const int j = 4 * q + e + f;
            const uint32_t bits = (__float_as_uint(f ? s2.y : s2.x) & ~31u) | j;
            const uint32_t key = rr[e + f] >= rho_i && j != self ? bits : 0xffffffffu;
            k2 = min(k2, max(k1, key));
            k1 = min(k1, key);
          }
        }
      }
      bool slow = false;
      if (need && k1 != 0xffffffffu) {
        const int j = k1 & 31u;
        float cj[N];
#pragma unroll
        for (int d = 0; d < N; ++d) cj[d] = reinterpret_cast<const float*>(s_blk[warp][d])[j];
        const float s = M::partial(x, cj, kp.mpar);
        if ((k2 >> 5) - (k1 >> 5) <= 1u)
          slow = __uint_as_float(k1 & ~31u) <= bnd;  // (the shortened value is not above the least)
        else if (s <= bnd) {
          if (reinterpret_cast<const float*>(s_blk[warp][N])[j] > rho_i && s * slack < s_best)
            take(j, s);
          else
            slow = true;
        }
      }
      nm = __ballot_sync(0xffffffffu, slow);
      if (nm) {
        const bool tied = TIE == CLUE_TIE_REFERENCE && slow && nh >= 0 && rank == rank_best &&
                          __uint_as_float(k1 & ~31u) >= s_best;
        nm = tie_block(nm, tied ? order_at(mq, nh) : -1, perm, order_at(mq, lane < cnt ? p0 + lane : p0), r, rho_i,
                       order_at(mq, h.p));
      }
    }
    while (nm) {
      const int hl = __ffs(nm) - 1;
      nm &= nm - 1;
      float xh[N], rho_h;
      smem_rec<N>(s_home[warp], hl, xh, rho_h);
      const float bnd_h = __shfl_sync(0xffffffffu, bnd, hl);
      const float s = M::partial(xh, c, kp.mpar);
      const bool ok = s <= bnd_h && r >= rho_h && p0 + lane != pw + hl;
      unsigned om = __ballot_sync(0xffffffffu, ok);
      if (om == 0) continue;
      if (om & (om - 1)) {
        // Of several, those that a strictly denser one is not strictly nearer than.  (The metric value is
        // negative for a negative weight: times slack would be nearer than itself.)
        const float near = warp_min_f(ok && r > rho_h ? s : INFINITY);
        om = __ballot_sync(0xffffffffu, ok && s <= fmaxf(near, near * slack));
      }
      if (om & (om - 1)) {  // still several
        om = tie_least<TIE>(om, s < 0.0f ? s : M::finish(s), r, rho_h, perm, order_at(mq, lane < cnt ? p0 + lane : p0),
                            order_at(mq, pw + hl));
        if (om == 0) continue;
      }
      const int j = __ffs(om) - 1;
      const float sj = __shfl_sync(0xffffffffu, s, j), rj = __shfl_sync(0xffffffffu, r, j);
      if (lane == hl) {
        if (rj > rho_i && sj * slack < s_best)
          take(j, sj);
        else
          consider(j, sj, rj);
      }
    }
  });
  // Seeds (KernelFindClusters) and every output but the label, while all of it is at hand.  d(i, nh)
  // is the nearest higher's distance, the same metric value bit for bit; without a nearest higher
  // the reference measures the distance to PointsView::operator[](-1), whose coordinates are
  // FLT_MAX (PointsCommon.hpp:75-81): an infinite or FLT_MAX distance, above any finite seed_dc,
  // which +inf decides the same way.
  const float dist = nh >= 0 ? M::finish(s_best) : INFINITY;
  const bool seed = valid && dist > kp.seed_dc && rho_i >= kp.rhoc;
  const int pos = order_at(mq, h.p);
  if (valid) {
    const int nhq = nh >= 0 ? order_at(mq, nh) : -1;
    sb.par[pos] = seed ? -1 : nhq;
    if (sb.nh) sb.nh[pos] = nhq;
    const int i = perm[pos];
    if (!dcheck_bad(st, i, kp.n, kChkSeedsPerm)) {
      if (seed) atomicOr(sb.bits + (i >> 5), 1u << (i & 31));
      if (out.is_seed) out.is_seed[i] = seed ? 1 : 0;
      if (out.rho) out.rho[i] = rho_i;
      if (out.nearest_higher)
        out.nearest_higher[i] = nhq >= 0 && !seed && !dcheck_bad(st, nhq, kp.n, kChkFinalizeNh) ? perm[nhq] : -1;
      if (out.delta) out.delta[i] = nh >= 0 ? dist : FLT_MAX;
    }
  }
  const uint32_t seeds = __ballot_sync(0xffffffffu, seed);
  if (seeds) {
    int first = 0;
    if (lane == 0) first = (int)atomicAdd(&st->n_seeds, (uint32_t)__popc(seeds));
    first = __shfl_sync(0xffffffffu, first, 0);
    if (seed) sb.list[first + __popc(seeds & ((1u << lane) - 1u))] = pos;
  }
  const uint32_t none = __ballot_sync(0xffffffffu, valid && nh < 0);
  if (lane == 0 && none) {
    atomicAdd(&st->seed_candidates, (uint32_t)__popc(none));
    atomicAdd(const_cast<uint32_t*>(&h.g->seed_candidates), (uint32_t)__popc(none));
  }
  // near-threshold decisions: densities within kNearTol of rhoc, distances of seed_dc or dm
  const uint32_t n_rhoc = __ballot_sync(0xffffffffu, valid && fabsf(rho_i - kp.rhoc) <= kNearTol * kp.rhoc);
  const uint32_t n_sdc =
      __ballot_sync(0xffffffffu, valid && nh >= 0 && fabsf(dist - kp.seed_dc) <= kNearTol * kp.seed_dc);
  const uint32_t n_dm = __ballot_sync(0xffffffffu, valid && nh >= 0 && fabsf(dist - kp.dm) <= kNearTol * kp.dm);
  if (lane == 0 && (n_rhoc | n_sdc | n_dm)) {
    if (n_rhoc) atomicAdd(&st->near_rhoc, (uint32_t)__popc(n_rhoc));
    if (n_sdc) atomicAdd(&st->near_seed_dc, (uint32_t)__popc(n_sdc));
    if (n_dm) atomicAdd(&st->near_dm, (uint32_t)__popc(n_dm));
  }
}

// Forms of the spatial-order density.  With unit amplitude the exponential kernel is
// exp2(kexp * d) and the zero-mean Gaussian exp2(kexp * d^2), kexp folding -avg or -1/(2 std^2)
// with log2(e); their value at d = 0 is exp2(0) = 1, the reference's self term, so no per-pair
// self test is needed.  Every other kernel takes the generic form.
enum { kDensGeneric = 0, kDensExpUnit = 1, kDensGauss0Unit = 2 };

// Local density over the Morton-ordered records (any order, kernels other than flat): the
// same candidate set as the reference (search-box tiles, d <= dc, self term 1), summed in
// spatial order.  Blocks farther than dc from every lane are skipped; inside a block, candidates
// that no lane of the warp holds within dc skip the kernel evaluation.
template <int N, int MT, int FORM>
__global__ void __launch_bounds__(kTileThreads, (N <= 4 ? 8 : 4) * 128 / kTileThreads) k_density_spatial(
    const KParams kp, Events ev, const int32_t* __restrict__ off, const int32_t* __restrict__ chunk_tile,
    const uint32_t* __restrict__ chunk_off, const uint32_t* __restrict__ chunk_total,
    const float4* __restrict__ rec_m,
    const int32_t* __restrict__ mq, const float4* __restrict__ blk, const float4* __restrict__ sblk,
    float4* __restrict__ rec_r, float kexp) {
  using M = Metric<N, MT>;
  __shared__ float4 s_rec[kTileThreads / 32][32 * Rec<N>::kWords];
  ChunkHome h;
  if (!chunk_home(kp, ev, off, chunk_tile, chunk_off, chunk_total, h)) return;
  const int pos = order_at(mq, h.p);
  const bool valid = h.valid;
  float x[N], wi;
  load_rec<N>(rec_m, h.p, x, wi);
  const int p_home = h.p;
  int hb[N], lo[N], hi[N];
  home_bins<N>(h.g, h.t, hb);
  lane_box<N>(kp, h.g, x, kp.dc, hb, lo, hi);
  if (!__any_sync(0xffffffffu, valid)) return;
  const float tdc = kp.t_dc;
  float4* sm = s_rec[threadIdx.x >> 5];
  float rho = 0.0f;
  spatial_sweep<N, M, false>(kp, h.g, off, hb, lo, hi, valid, x, blk, sblk, -INFINITY, p_home, [&]() { return tdc; },
                      [&](int p0, int p1, bool need, int64_t) {
    const int cnt = p1 - p0;
    stage_block<N>(sm, rec_m, p0, cnt);
    const int jself = p_home - p0;
    auto pair = [&](int j, bool in_block) {
      float c[N], wj;
      smem_rec<N>(sm, j, c, wj);
      const float s = M::partial(x, c, kp.mpar);
      const bool in = need && in_block && s <= tdc;
      if (__any_sync(0xffffffffu, in)) {
        float kv;
        if (FORM == kDensExpUnit) {
          kv = ex2_approx(kexp * (M::kRoot ? sqrt_approx(s) : s));
        } else if (FORM == kDensGauss0Unit) {
          kv = ex2_approx(kexp * (M::kRoot ? s : s * s));
        } else {
          const float dist = M::kRoot ? sqrt_approx(s) : s;
          kv = (j == jself) ? 1.0f : kernel_value_fast(kp.kernel_type, kp.kpar, kp.ginv, dist);
        }
        const float t = kv * wj;
        if (in) rho = fadd(rho, t);
      }
    };
    int j0 = 0;
    for (; j0 + 8 <= cnt; j0 += 8) {
#pragma unroll
      for (int u = 0; u < 8; ++u) pair(j0 + u, true);
    }
    if (j0 < cnt) {
#pragma unroll
      for (int u = 0; u < 8; ++u) pair(j0 + u, j0 + u < cnt);
    }
  });
  if (valid) store_rec<N>(rec_r, pos, x, rho);
}

// ---- symmetric spatial density -------------------------------------------------
// For metrics whose value bounds every coordinate difference (Euclidean, Manhattan, Chebyshev)
// and no wrapped coordinate, d(i, j) <= dc already places j's tile inside i's search box, so the
// candidate set is {j : d(i, j) <= dc} and every pair can be evaluated once for both points.
// Blocks are 32 consecutive Morton-ordered records counted from their tile's start (so the
// result does not depend on where a tile lies in a batch): block slot 4 c + w is warp w of
// chunk c.  The warp of block A evaluates A against itself one-sidedly and every block B of its
// tile after A and of the later tiles of its search-box union both ways: at step k lane l reads
// candidate l ^ k from shared memory, adds K(d) w_j to its own sum and hands K(d) w_i to the
// candidate's lane by shuffle; that lane's sum is then added in fixed point (exact integer adds, so
// the order of arrival does not matter) to the candidate's accumulator.

// Block boxes in compact order: block b of tile u is entry bo[u] + b (bo = exclusive scan of
// the tiles' block counts).  One thread per (chunk, warp) slot; slots past a tile's end write
// nothing.
template <int N>
__global__ void __launch_bounds__(256) k_tblock_bbox(int max_slots, const uint32_t* __restrict__ chunk_total,
                                                    const int32_t* __restrict__ off,
                                                    const int32_t* __restrict__ chunk_tile,
                                                    const uint32_t* __restrict__ chunk_off,
                                                    const uint32_t* __restrict__ bo,
                                                    const float4* __restrict__ rec_m, float4* __restrict__ tblk) {
  constexpr int BW = Blk<N>::kWords;
  const int nslots = min(max_slots, kChunkWarps * (int)*chunk_total);
  const int stride = gridDim.x * blockDim.x;
  for (int sl = blockIdx.x * blockDim.x + threadIdx.x; sl < nslots; sl += stride) {
    const int c = sl / kChunkWarps;
    const int t = chunk_tile[c];
    const int b = (c - (int)chunk_off[t]) * kChunkWarps + sl % kChunkWarps;
    const int first = off[t] + (b << 5);
    const int cnt = min(32, off[t + 1] - first);
    if (cnt <= 0) continue;
    float bb[4 * BW];
#pragma unroll
    for (int d = 0; d < N; ++d) {
      bb[d] = INFINITY;
      bb[N + d] = -INFINITY;
    }
#pragma unroll
    for (int k = 2 * N; k < 4 * BW; ++k) bb[k] = 0.0f;
    for (int r = 0; r < cnt; ++r) {
      float x[N], pl;
      load_rec<N>(rec_m, first + r, x, pl);
#pragma unroll
      for (int d = 0; d < N; ++d) {
        bb[d] = fminf(bb[d], x[d]);
        bb[N + d] = fmaxf(bb[N + d], x[d]);
      }
    }
    const size_t id = (size_t)bo[t] + b;
#pragma unroll
    for (int k = 0; k < BW; ++k)
      tblk[id * BW + k] = make_float4(bb[4 * k], bb[4 * k + 1], bb[4 * k + 2], bb[4 * k + 3]);
  }
}

// Fixed-point exponent of an event: contributions times 2^F stay below 2^61 in total
// (|sum| <= count * max|w| * max kernel value).
__device__ __forceinline__ int fix_exponent(const EvGrid* g, float kmax) {
  const float bound = __uint_as_float(g->wmax_bits) * (float)g->pt_count * kmax;
  int e = 0;
  frexpf(bound, &e);  // bound < 2^e
  return max(-126, min(126, 61 - e));
}

// A candidate block in shared memory for the pair steps, in pairs of neighbours: component j (N: the
// weight) of candidates 2 m and 2 m + 1 side by side, two components to a 16-byte word, 16 words (one
// per pair) in a row, so that two steps read both candidates of a pair as operands of paired
// arithmetic, without a move.  Two neighbouring lanes read the same words.
// The sweep is bound by the MUFU pipe (two operations a pair for the exponential kernel, 73% busy) and
// instruction issue (71%).  With every component by butterfly shuffle (eight shuffles for two steps,
// the shared-memory pipe 75% busy as well, and moves to pair the operands) it took 7000 instructions
// a warp, now 4700: 3.43 -> 3.22 ms on the 4096-event batch, 1.16 -> 1.01 ms on 4M 3-D points, 0.30 ->
// 0.27 ms on 1M 2-D points (Gaussian).  A second copy for odd lanes, which spares the two selects a
// step pair, costs more in shared-memory reads: 3.53 and 1.12 ms.
template <int N>
struct PairSmem {
  static constexpr int kRows = (N + 2) / 2;
  static constexpr int kFloats = kRows * 64;
};
// All components of a pair at shared-memory address `a` (row 0's word); "memory", since ordinary stores
// of the warp put them there.
template <int N>
__device__ __forceinline__ void load_pairs(uint32_t a, unsigned long long* c) {
#pragma unroll
  for (int f = 0; f < (N + 1) / 2; ++f)
    asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(c[2 * f]), "=l"(c[2 * f + 1]) : "r"(a + 256u * f) : "memory");
  if constexpr ((N + 1) & 1) asm volatile("ld.shared.u64 %0, [%1];" : "=l"(c[N]) : "r"(a + 256u * (N / 2)) : "memory");
}

// VAR selects measured alternatives of the pair step (clue_tuning.density_gate / density_exp2):
// bit 0: a warp vote per pair of steps skips the kernel evaluation and the mirrored shuffles when
// no lane of the warp has a candidate within dc (the same bits: the skipped terms are zeros);
// bit 1: the unit-amplitude forms evaluate 2^x with exp2_poly2 on the FMA pipe instead of
// ex2.approx on the MUFU pipe (within 5e-7 relative per term).
template <int N, int MT, int FORM, int VAR>
__global__ void __launch_bounds__(kTileThreads, (N <= 4 ? 8 : 4) * 128 / kTileThreads) k_density_sym(
    const KParams kp, Events ev, const int32_t* __restrict__ off, const int32_t* __restrict__ chunk_tile,
    const uint32_t* __restrict__ chunk_off, const uint32_t* __restrict__ chunk_total,
    const float4* __restrict__ rec_m, const int32_t* __restrict__ mq, const uint32_t* __restrict__ bo,
    const float4* __restrict__ tblk, float4* __restrict__ rec_r, int64_t* __restrict__ rho_fix, float kexp,
    float kmax, DevStatus* st) {
  using M = Metric<N, MT>;
  constexpr int BW = Blk<N>::kWords;
  __shared__ float4 s_rec[kTileThreads / 32][32 * Rec<N>::kWords];
  __shared__ alignas(256) float4 s_pair[kTileThreads / 32][PairSmem<N>::kFloats / 4];
  const int c = blockIdx.x;
  if (c >= (int)*chunk_total) return;
  const int lane = lane_id(), warp = threadIdx.x >> 5;
  float* sp = reinterpret_cast<float*>(s_pair[warp]);
  const uint32_t sp_own = (uint32_t)__cvta_generic_to_shared(sp) + 16u * (lane >> 1);
  const bool odd = lane & 1;
  const int t = chunk_tile[c];
  if (t < 0) return;  // a slot that its event does not need (k_build)
  const int a_loc = (c - (int)chunk_off[t]) * kChunkWarps + warp;  // block of the tile
  const int startA = off[t] + (a_loc << 5);
  const int cntA = min(32, off[t + 1] - startA);
  if (cntA <= 0) return;  // whole warp: this block of the chunk is past the tile's end
  const EvGrid* g = ev.eg + event_of(ev.pt, ev.chunk_ev, kp.n_events, off[t]);
  const bool hv = lane < cntA;
  const int pA = startA + (hv ? lane : 0);
  float x[N], wi;
  load_rec<N>(rec_m, pA, x, wi);
  int hb[N], lo[N], hi[N];
  home_bins<N>(g, t, hb);
  lane_box<N>(kp, g, x, kp.dc, hb, lo, hi);
  int wl[N], wh[N];
#pragma unroll
  for (int d = 0; d < N; ++d) {
    wl[d] = warp_min_i(hv ? lo[d] : INT_MAX);
    wh[d] = warp_max_i(hv ? hi[d] : INT_MIN);
  }
  const float tdc = kp.t_dc, thr = hv ? tdc : -INFINITY;
  float hlo[N], hhi[N];  // box of block A
  unsigned long long x2[N];
#pragma unroll
  for (int d = 0; d < N; ++d) {
    hlo[d] = warp_min_f(hv ? x[d] : INFINITY);
    hhi[d] = warp_max_f(hv ? x[d] : -INFINITY);
    x2[d] = pk2(make_float2(x[d], x[d]));
  }
  const unsigned long long one = pk2(make_float2(kp.one, kp.one));
  const float scale = ldexpf(1.0f, fix_exponent(g, kmax));
  auto kval = [&](float s, bool self) -> float {
    if (FORM == kDensExpUnit) return ex2_approx(kexp * (M::kRoot ? sqrt_approx(s) : s));
    if (FORM == kDensGauss0Unit) return ex2_approx(kexp * (M::kRoot ? s : s * s));
    const float dist = M::kRoot ? sqrt_approx(s) : s;
    return self ? 1.0f : kernel_value_fast(kp.kernel_type, kp.kpar, kp.ginv, dist);
  };
  const float2 kexp2 = make_float2(kexp, kexp);
  auto kval2 = [&](float2 s) -> float2 {
    if (FORM == kDensExpUnit) {
      const float2 d = M::kRoot ? make_float2(sqrt_approx(s.x), sqrt_approx(s.y)) : s;
      const float2 e = mul2(kexp2, d);
      if (VAR & 2) return exp2_poly2(e);
      return make_float2(ex2_approx(e.x), ex2_approx(e.y));
    }
    if (FORM == kDensGauss0Unit) {
      const float2 e = mul2(kexp2, M::kRoot ? s : mul2(s, s));
      if (VAR & 2) return exp2_poly2(e);
      return make_float2(ex2_approx(e.x), ex2_approx(e.y));
    }
    return make_float2(kval(s.x, false), kval(s.y, false));
  };
  float acc = 0.0f;
  // block A against itself, one-sided (the self pair gives the reference's self term)
  {
    float4* sm = s_rec[warp];
    stage_block<N>(sm, rec_m, startA, cntA);
    if (FORM == kDensGeneric) {  // the generic kernel needs the self test
      for (int j = 0; j < cntA; ++j) {
        float cx[N], wj;
        smem_rec<N>(sm, j, cx, wj);
        const float sd = M::partial(x, cx, kp.mpar);
        const bool in = hv && sd <= tdc;
        if (__any_sync(0xffffffffu, in)) {
          const float t2 = kval(sd, j == lane) * wj;
          if (in) acc = fadd(acc, t2);
        }
      }
    } else {
      // two candidates at a time, no branch (the own block almost always has pairs within dc);
      // a record past the block's end (stale shared memory) is masked with its weight
      float2 acc2 = make_float2(0.0f, 0.0f);
      for (int j = 0; j < cntA; j += 2) {
        float ca[N], cb[N], wa, wb;
        smem_rec<N>(sm, j, ca, wa);
        smem_rec<N>(sm, j + 1, cb, wb);
        const bool bv = j + 1 < cntA;
        const float2 sd = partial_pair<N, MT>(x, ca, cb, kp.mpar);
        float2 kv = kval2(sd);
        kv.x = hv && sd.x <= tdc ? kv.x : 0.0f;
        kv.y = hv && bv && sd.y <= tdc ? kv.y : 0.0f;
        acc2 = fma2(kv, make_float2(wa, bv ? wb : 0.0f), acc2);
      }
      acc = fadd(acc, fadd(acc2.x, acc2.y));
    }
  }
  // later blocks of the own tile, then the later tiles of the union box, both ways
  int v[N];
#pragma unroll
  for (int d = 0; d < N; ++d) v[d] = wl[d];
  while (true) {
    int u = g->tile_base;
#pragma unroll
    for (int d = 0; d < N; ++d) u += g->stride[d] * v[d];
    if (u >= t && !dcheck_bad(st, u, kp.ntiles, kChkDensityTile)) {
      const int pb = off[u], pe = off[u + 1];
      const int nb = (pe - pb + 31) >> 5;
      const int b0 = u == t ? a_loc + 1 : 0, box0 = (int)bo[u];
      // the block boxes are tested 32 at a time against the box of block A, and those in reach by
      // every lane for its own point
      for (int c0 = b0; c0 < nb; c0 += 32) {
        bool near = false;
        if (c0 + lane < nb) {
          float bb[4 * BW];
          load_box<N>(tblk, box0 + c0 + lane, bb);
          near = lower_box<N, M>(hlo, hhi, bb, bb + N, kp.mpar) <= tdc;
        }
        for (unsigned mask = __ballot_sync(0xffffffffu, near); mask; mask &= mask - 1) {
          const int b = c0 + __ffs(mask) - 1;
          float bb[4 * BW];
          load_box<N>(tblk, box0 + b, bb);
          const bool need = hv && lower_point<N, M>(x, bb, bb + N, kp.mpar) <= tdc;
          if (!__any_sync(0xffffffffu, need)) continue;
          const int first = pb + (b << 5);
          const int cntB = min(32, pe - first);
          const bool cv = lane < cntB;
          // lane m owns candidate m of the block; at step k lane l meets candidate l ^ k and the
          // candidate's owner collects the term from lane m ^ k = l (shuffles with immediate lane
          // masks), so no value is carried from one step to the next; the candidates themselves are
          // read from shared memory, two steps at a time (PairSmem)
          {
            float ox[N + 1];
            load_rec<N>(rec_m, first + (cv ? lane : 0), ox, ox[N]);
            if (!cv) {
#pragma unroll
              for (int d = 0; d < N; ++d) ox[d] = INFINITY;  // never within dc
              ox[N] = 0.0f;
            }
            __syncwarp();  // the previous block's readers are done
#pragma unroll
            for (int j = 0; j <= N; ++j) {
              sp[(j / 2) * 64 + (lane >> 1) * 4 + (j & 1) * 2 + (lane & 1)] = ox[j];
            }
            __syncwarp();
          }
          // two steps at a time, with paired arithmetic; the own terms of this block are summed
          // (fused multiply-add) in two running sums, even and odd steps (in the other order in odd
          // lanes, which meet a pair's second candidate first), added at the block's end
          float2 acc2 = make_float2(0.0f, 0.0f), cacc2 = make_float2(0.0f, 0.0f);
          const float2 wi2 = make_float2(wi, wi);
#pragma unroll
          for (int k = 0; k < 32; k += 2) {
            unsigned long long c2[N + 1];
            load_pairs<N>(sp_own ^ (uint32_t)(8 * k), c2);
            const float2 cw = upk2(c2[N]);
            const float2 sd = partial_packed<N, MT>(x2, c2, kp.mpar, one);
            const bool ix = sd.x <= thr, iy = sd.y <= thr;
            if ((VAR & 1) == 0 || __any_sync(0xffffffffu, ix || iy)) {
              float2 kv;
              if constexpr (FORM == kDensGeneric || (VAR & 2) != 0) {
                kv = kval2(sd);
                kv.x = ix ? kv.x : 0.0f;
                kv.y = iy ? kv.y : 0.0f;
              } else {
                kv = kernel_within<FORM == kDensExpUnit, M::kRoot>(sd, thr, kexp2);
              }
              acc2 = fma2(kv, cw, acc2);
              const float2 tc = mul2(kv, wi2);
              const float t0 = odd ? tc.y : tc.x, t1 = odd ? tc.x : tc.y;  // of steps k and k + 1
              cacc2 = add2(cacc2, make_float2(__shfl_xor_sync(0xffffffffu, t0, k), __shfl_xor_sync(0xffffffffu, t1, k + 1)));
            }
          }
          acc = fadd(acc, fadd(acc2.x, acc2.y));
          const float cacc = fadd(cacc2.x, cacc2.y);
          if (cv && cacc != 0.0f) {
            const int mi = order_at(mq, first + lane);
            if (!dcheck_bad(st, mi, kp.n, kChkDensityMirror))
              atomicAdd(reinterpret_cast<unsigned long long*>(rho_fix + mi), (unsigned long long)__float2ll_rn(cacc * scale));
          }
        }
      }
    }
    int d = N - 1;
    for (; d >= 0; --d) {
      if (v[d] < wh[d]) {
        ++v[d];
        break;
      }
      v[d] = wl[d];
    }
    if (d < 0) break;
  }
  if (hv) store_rec<N>(rec_r, order_at(mq, pA), x, acc);
}

// rho = own-side sum + the fixed-point sum of the contributions received as a candidate.
template <int N>
__global__ void __launch_bounds__(256) k_density_combine(const KParams kp, Events ev, int n,
                                                         const int64_t* __restrict__ rho_fix,
                                                         float4* __restrict__ rec_r, float kmax) {
  const int stride = gridDim.x * blockDim.x;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += stride) {
    bool uniform;
    const EvGrid* g = ev.eg + warp_event(ev.pt, ev.chunk_ev, kp.n_events, q, true, uniform);
    float x[N], acc;
    load_rec<N>(rec_r, q, x, acc);
    const float recv = (float)((double)rho_fix[q] * ldexp(1.0, -fix_exponent(g, kmax)));
    store_rec<N>(rec_r, q, x, fadd(acc, recv));
  }
}

// Boxes (and largest payloads) of every block of 32 and every super-block of 1024 Morton-ordered
// records, one CTA per super-block.  GATHER takes the records through the order mq into rec_m
// first; otherwise rec is in Morton order (a composite sort) and its densities get the symmetric
// sweep's fixed-point sums added in (as k_density_combine does).
template <int N, bool GATHER>
__global__ void __launch_bounds__(1024) k_boxes(const KParams kp, Events ev, const int32_t* __restrict__ mq,
                                                float4* rec, float4* __restrict__ rec_m,
                                                const int64_t* __restrict__ rho_fix, float kmax,
                                                float4* __restrict__ blk, float4* __restrict__ sblk) {
  constexpr int BW = Blk<N>::kWords;
  __shared__ float s_box[32][2 * N + 1];
  const int lane = lane_id(), warp = threadIdx.x >> 5, n = kp.n;
  const int b = blockIdx.x * 32 + warp, nblk = (n + 31) >> 5;
  if (b < nblk) {
    const int q = (b << 5) + lane;
    const bool valid = q < n;
    // lanes past the end repeat the last record: warp_event takes the last lane's for the largest
    const int qq = min(q, n - 1);
    float x[N], pl;
    if (GATHER) {
      load_rec<N>(rec, mq[qq], x, pl);
      if (valid) store_rec<N>(rec_m, q, x, pl);
    } else {
      bool uniform;
      const EvGrid* g = ev.eg + warp_event(ev.pt, ev.chunk_ev, kp.n_events, qq, true, uniform);
      load_rec<N>(rec, qq, x, pl);
      pl = fadd(pl, (float)((double)rho_fix[qq] * ldexp(1.0, -fix_exponent(g, kmax))));
      if (valid) store_rec<N>(rec, q, x, pl);
    }
    write_block_box<N>(blk, b, x, pl);
    float lo[N], hi[N];
#pragma unroll
    for (int d = 0; d < N; ++d) {
      lo[d] = warp_min_f(x[d]);
      hi[d] = warp_max_f(x[d]);
    }
    pl = warp_max_f(pl);
    if (lane == 0) {
#pragma unroll
      for (int d = 0; d < N; ++d) {
        s_box[warp][d] = lo[d];
        s_box[warp][N + d] = hi[d];
      }
      s_box[warp][2 * N] = pl;
    }
  }
  __syncthreads();
  if (warp == 0) {
    const int w = min(lane, nblk - 1 - (int)blockIdx.x * 32);  // blocks past the end repeat the last one
    float v[4 * BW];
#pragma unroll
    for (int k = 0; k < 4 * BW; ++k) v[k] = 0.0f;
#pragma unroll
    for (int d = 0; d < N; ++d) {
      v[d] = warp_min_f(s_box[w][d]);
      v[N + d] = warp_max_f(s_box[w][N + d]);
    }
    v[2 * N] = warp_max_f(s_box[w][2 * N]);
    if (lane < BW) {
      float4 out;
#pragma unroll
      for (int k = 0; k < BW; ++k)
        if (k == lane) out = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
      sblk[(size_t)blockIdx.x * BW + lane] = out;
    }
  }
}

// Near-tie count of the nearest-higher stage (CLUE_FLAG_NEAR_TIES), after k_nearest_higher:
// a point counts when its chosen nearest higher, or a candidate of its search box at most as
// far as that one (within dm when none was found) that is not its own record, has a density
// within kNearTol of the point's own.  These are the points whose nearest higher can change
// when densities move by that much (ClusteringKernels.hpp:129-143).  A pruned sweep like
// nearest higher's: blocks beyond the chosen distance, or whose densities all lie below
// rho_i - tol |rho_i|, are skipped.
template <int N, int MT>
__global__ void __launch_bounds__(kTileThreads) k_near_ties(
    const KParams kp, Events ev, const int32_t* __restrict__ off,
    const int32_t* __restrict__ chunk_tile, const uint32_t* __restrict__ chunk_off,
    const uint32_t* __restrict__ chunk_total, const float4* __restrict__ rec_r, const float4* __restrict__ rec_m,
    const int32_t* __restrict__ mq, const float4* __restrict__ blk, const float4* __restrict__ sblk,
    const int32_t* __restrict__ nh_s, DevStatus* st) {
  using M = Metric<N, MT>;
  ChunkHome h;
  if (!chunk_home(kp, ev, off, chunk_tile, chunk_off, chunk_total, h)) return;
  const int pos = order_at(mq, h.p);
  const bool valid = h.valid;
  float x[N], rho_i;
  load_rec<N>(rec_r, pos, x, rho_i);
  int hb[N], lo[N], hi[N];
  home_bins<N>(h.g, h.t, hb);
  lane_box<N>(kp, h.g, x, kp.dm, hb, lo, hi);
  if (!__any_sync(0xffffffffu, valid)) return;
  __shared__ float4 s_rec[kTileThreads / 32][32 * Rec<N>::kWords];
  __shared__ int32_t s_q[kTileThreads / 32][32];
  float4* sm = s_rec[threadIdx.x >> 5];
  int32_t* sq = s_q[threadIdx.x >> 5];
  auto near = [&](float r) {
    const float m = fmaxf(fabsf(r), fabsf(rho_i));
    return m > 0.0f && fabsf(r - rho_i) <= kNearTol * m;
  };
  const int nh = nh_s[pos];
  float bnd = kp.t_dm;
  bool flag = false;
  if (nh >= 0) {
    float c[N], rho_nh;
    load_rec<N>(rec_r, nh, c, rho_nh);
    bnd = M::partial(x, c, kp.mpar);
    flag = near(rho_nh);
  }
  const float pmin = rho_i - kNearTol * fabsf(rho_i);
  spatial_sweep<N, M, false>(kp, h.g, off, hb, lo, hi, valid, x, blk, sblk, pmin, h.p, [&]() { return bnd; },
                             [&](int p0, int p1, bool need, int64_t) {
    const int cnt = p1 - p0;
    stage_block<N>(sm, rec_m, p0, cnt, sq, mq);
    for (int j = 0; j < cnt; ++j) {
      float c[N], rj;
      smem_rec<N>(sm, j, c, rj);
      const float s = M::partial(x, c, kp.mpar);
      flag = flag || (need && s <= bnd && sq[j] != pos && near(rj));
    }
  });
  const uint32_t cnt_w = __ballot_sync(0xffffffffu, valid && flag);
  if ((threadIdx.x & 31) == 0 && cnt_w) atomicAdd(&st->nh_near_ties, (uint32_t)__popc(cnt_w));
}

// Seed list capacity of an event: every seed, or the reference's SeedArray capacity
// max(seed_capacity, points without nearest higher) (SetupSeeds.hpp:10-20).
__device__ __forceinline__ int64_t seed_cap(const KParams& kp, const EvGrid* g) {
  if (kp.seed_capacity < 0) return INT64_MAX;
  return kp.seed_capacity > (int64_t)g->seed_candidates ? kp.seed_capacity : (int64_t)g->seed_candidates;
}

// ---- stage 5: labels ---------------------------------------------------------
// The parents form a forest over the tile-sorted positions.  A root has a negative parent: -1 (no
// label: a point without nearest higher that is not a seed, or a seed beyond the capacity) or
// -2 - label.
// Bound by memory: the nearest-higher search writes everything but the labels while its own work
// hides the scatter, seeds are ranked by a scan over one bit per point, and a point reads its parent
// chain and its index and writes its label.  A pass for the seeds with a flag word per point, its
// scan, four jump launches and an output pass over all arrays took 0.605 ms on the 4096-event batch
// and 0.253 ms on 4M 3-D points; this takes 0.17 and 0.071 ms, and 0.10 ms and 0.02 ms more in the
// search.

// Seeds before point i of the original order.
__device__ __forceinline__ uint32_t seed_rank_of(const uint32_t* bits, const uint32_t* rank,
                                                 int i) {
  return rank[i >> 5] + (uint32_t)__popc(bits[i >> 5] & ((1u << (i & 31)) - 1u));
}

// The label of every seed (its rank by index inside its event) written as its root value, and per
// event the seeds and clusters (optional outputs) with their total in st->n_clusters.
__device__ __forceinline__ void seed_labels(const KParams& kp, Events ev, const uint32_t* bits, const uint32_t* rank,
                                            const uint32_t* total, const int32_t* list, const int32_t* perm,
                                            int32_t* par, int32_t* n_seeds, int32_t* n_clusters, DevStatus* st) {
  const int stride = gridDim.x * blockDim.x, first = blockIdx.x * blockDim.x + threadIdx.x;
  const int ns = (int)st->n_seeds;
  for (int k = first; k < ns; k += stride) {
    const int pos = list[k], i = perm[pos];
    if (dcheck_bad(st, i, kp.n, kChkFinalizeRoot)) continue;
    const int e = event_of(ev.pt, ev.chunk_ev, kp.n_events, pos);
    const uint32_t lab = seed_rank_of(bits, rank, i) - seed_rank_of(bits, rank, ev.pt[e]);
    if ((int64_t)lab < seed_cap(kp, ev.eg + e)) par[pos] = -2 - (int)lab;
  }
  for (int e = first; e < kp.n_events; e += stride) {
    const uint32_t a = seed_rank_of(bits, rank, ev.pt[e]);
    const uint32_t b = e + 1 < kp.n_events ? seed_rank_of(bits, rank, ev.pt[e + 1]) : *total;
    const int64_t seeds = (int64_t)(b - a), cap = seed_cap(kp, ev.eg + e);
    const int64_t nc = seeds < cap ? seeds : cap;
    if (n_seeds) n_seeds[e] = (int32_t)seeds;
    if (n_clusters) n_clusters[e] = (int32_t)nc;
    atomicAdd(&st->n_clusters, (uint32_t)nc);
  }
}

__global__ void __launch_bounds__(256) k_seed_labels(const KParams kp, Events ev, const uint32_t* __restrict__ bits,
                                                     const uint32_t* __restrict__ rank,
                                                     const uint32_t* __restrict__ total,
                                                     const int32_t* __restrict__ list,
                                                     const int32_t* __restrict__ perm, int32_t* __restrict__ par,
                                                     int32_t* __restrict__ n_seeds, int32_t* __restrict__ n_clusters,
                                                     DevStatus* st) {
  seed_labels(kp, ev, bits, rank, total, list, perm, par, n_seeds, n_clusters, st);
}

// The same behind a scan of the seed bits, for calls of up to kScanOneBlock words (a launch less): every
// block scans all of them for itself into shared memory and takes its share of the seeds and events.
__global__ void __launch_bounds__(1024) k_seed_labels_scan(const KParams kp, Events ev, const uint32_t* bits,
                                                           uint32_t* total, int words, const int32_t* list,
                                                           const int32_t* perm, int32_t* par, int32_t* n_seeds,
                                                           int32_t* n_clusters, DevStatus* st) {
  constexpr int kPer = (int)(kScanOneBlock / 1024);
  __shared__ uint32_t s_scan[33], s_total, rank[kScanOneBlock];
  const int base = threadIdx.x * kPer;
  uint32_t c[kPer], sum = 0;
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    c[k] = base + k < words ? (uint32_t)__popc(bits[base + k]) : 0u;
    sum += c[k];
  }
  uint32_t all, run = build_scan<32>(s_scan, sum, threadIdx.x & 31, threadIdx.x >> 5, &all);
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    if (base + k < words) rank[base + k] = run;
    run += c[k];
  }
  if (threadIdx.x == 0) s_total = all;
  if (blockIdx.x == 0 && threadIdx.x == 0) *total = all;
  __syncthreads();
  seed_labels(kp, ev, bits, rank, &s_total, list, perm, par, n_seeds, n_clusters, st);
}

// Blocks of k_seed_labels_scan: one for every 4096 points.  One alone takes 0.8 us for every 1024 seeds
// (label stage of 262144 seeds 202 us, 17 with 64 blocks; of 246 seeds 17 and 13 us; separate scans 54).
constexpr int kSeedBlockPoints = 4096, kSeedBlocks = 64;

// Pointer jumping on the forest: every parent pointer is replaced by its grandparent until it
// names a root.  All writes move a pointer to an ancestor, so concurrent updates are safe.
// With LABELS every point that reaches its root gets its label.
// A thread makes up to `passes` passes over its chains, at most `hops` jumps a chain in each.  The grid
// is one that the GPU holds at once (label_blocks), so the chains of all points move on together and a
// pass finds the parents of the one before far ahead.  A chain climbed to its end at once goes point by
// point through those whose threads have not begun: a ramp of 1M points took 16.2 ms with up to 4096 jumps
// at once, 0.06 with 16 a pass (8: 0.06, 32: 0.17, 64: 0.42), one of 4M points 13 and 0.15 ms.  What is
// unresolved after the last pass is recorded in st->unresolved[round] and left to the next launch.
struct JumpLimits {
  int hops, passes;
};
template <bool LABELS, int K>
__device__ __forceinline__ void jump(int32_t* par, const int32_t* __restrict__ perm, int32_t* __restrict__ label,
                                     int n, JumpLimits limits, DevStatus* st, int round) {
  const int stride = gridDim.x * blockDim.x;
  uint32_t todo = ~0u;  // groups of K chains with an unresolved one (the last bit: of all from the 32nd on)
  for (int pass = 0; pass < limits.passes && todo; ++pass) {
    uint32_t left = 0, bit = 1u;
    // K chains per thread walked in lockstep: each step's parent loads are independent, so they are in
    // flight together (the walk is bound by load latency, not bandwidth)
    for (int64_t pos0 = blockIdx.x * blockDim.x + threadIdx.x; pos0 < n; pos0 += (int64_t)K * stride) {
      const uint32_t group = bit;
      if (bit != 0x80000000u) bit <<= 1;
      if (!(todo & group)) continue;
      int p[K], i[K];
      bool act[K];
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int64_t pos = pos0 + (int64_t)k * stride;
        p[k] = pos < n ? par[pos] : -1;
        if (LABELS) i[k] = pos < n ? perm[pos] : -1;
        act[k] = p[k] >= 0;
      }
      for (int it = 0; it < limits.hops; ++it) {
        bool any = false;
#pragma unroll
        for (int k = 0; k < K; ++k) {
          if (act[k] && dcheck_bad(st, p[k], n, kChkJumpParent)) act[k] = false;
          if (act[k]) {
            const int pp = __ldcg(par + p[k]);
            if (pp < 0) {
              act[k] = false;
              if (LABELS) p[k] = pp;  // the root's value
            } else {
              p[k] = pp;
              par[pos0 + (int64_t)k * stride] = pp;
            }
          }
          any |= act[k];
        }
        if (!any) break;
      }
#pragma unroll
      for (int k = 0; k < K; ++k) {
        if (act[k]) {  // still climbing after the pass's jumps
          const int pp = __ldcg(par + p[k]);
          if (pp >= 0)
            left |= group;
          else if (LABELS)
            p[k] = pp;
        }
        if (LABELS && p[k] < 0 && i[k] >= 0) label[i[k]] = p[k] < -1 ? -2 - p[k] : -1;
      }
    }
    todo = left;
  }
  if (__any_sync(0xffffffffu, todo != 0) && (threadIdx.x & 31) == 0) atomicAdd(&st->unresolved[round], 1u);
  if (blockIdx.x == 0 && threadIdx.x == 0) atomicMax(&st->label_rounds, (uint32_t)round + 1);
}

// First round: the climb that ends most chains writes the labels as well.  Four chains per thread from
// 2M points on, one below, where there are threads enough (label stage: 4M points 0.075 ms against
// 0.091 with one; 1M points 0.056 ms with four, 0.048 with one).  Eight blocks an SM, so that the grid of
// label_blocks is resident: the 4096-event batch's label stage 0.200 -> 0.169 ms, 4M points 0.075 -> 0.071 (two
// chains 0.194 and 0.073, three 0.177 and 0.071; five blocks of 40 registers 0.212 and 0.081).
constexpr int kLabelChainPoints = 1 << 21;
template <int K>
__global__ void __launch_bounds__(256, 8) k_labels(int32_t* par, const int32_t* __restrict__ perm,
                                                int32_t* __restrict__ label, int n, JumpLimits limits, int rounds,
                                                DevStatus* st) {
  if (blockIdx.x == 0 && threadIdx.x == 0) st->label_enqueued = (uint32_t)rounds;
  jump<true, K>(par, perm, label, n, limits, st, 0);
}

__global__ void __launch_bounds__(256, 8) k_jump(int32_t* par, int n, JumpLimits limits, DevStatus* st, int round) {
  if (st->unresolved[round - 1] == 0) return;
  jump<false, 4>(par, nullptr, nullptr, n, limits, st, round);
}

// All labels again, from parents that name roots, when the first round left a chain unresolved.
// `rounds` have been enqueued by now (a blocking call's host adds to the one of k_labels), so a status
// read after this call finds the last one's outcome.
__global__ void __launch_bounds__(256) k_labels_again(const int32_t* __restrict__ par,
                                                      const int32_t* __restrict__ perm, int32_t* __restrict__ label,
                                                      int n, int rounds, DevStatus* st) {
  if (blockIdx.x == 0 && threadIdx.x == 0) st->label_enqueued = (uint32_t)rounds;
  if (st->unresolved[0] == 0) return;
  const int stride = gridDim.x * blockDim.x;
  for (int pos = blockIdx.x * blockDim.x + threadIdx.x; pos < n; pos += stride) {
    int p = par[pos];
    if (p >= 0 && dcheck_bad(st, p, n, kChkFinalizeRoot)) continue;
    if (p >= 0) p = par[p];
    const int i = perm[pos];
    if (!dcheck_bad(st, i, n, kChkFinalizeRoot)) label[i] = p < -1 ? -2 - p : -1;
  }
}

// ---- stage 5, breadth-first form (clue_tuning.labels_bfs) ----------------------
// The reference's follower association map (Followers::fill, AssociationMap.hpp:193-251: counts
// per nearest higher, a scan, a scatter) and its assignment from the seeds
// (KernelAssignClusters, ClusteringKernels.hpp:246-281, a depth-first walk per seed), here with
// the walk done level by level over all seeds at once: the frontier of level l holds the points
// l steps below a seed, and each of their followers takes the seed as its parent.  Points no
// seed reaches keep their nearest higher as parent, whose chain ends at a point that is not a
// seed, so k_labels gives them -1 as pointer jumping does; a frontier left over after the last
// enqueued level is climbed there too.

// counts[p] = followers of p (par[i] = p >= 0).
__global__ void __launch_bounds__(256) k_follower_count(const int32_t* __restrict__ par, int n,
                                                        uint32_t* __restrict__ counts) {
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const int p = par[i];
    if (p >= 0) atomicAdd(counts + p, 1u);
  }
}

// Scatter of every follower into its parent's run (order inside a run is the atomic order; the
// labels do not depend on it).  cursor starts as the exclusive scan of the counts.
__global__ void __launch_bounds__(256) k_follower_fill(const int32_t* __restrict__ par, int n,
                                                       uint32_t* __restrict__ cursor, int32_t* __restrict__ followers) {
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const int p = par[i];
    if (p >= 0) followers[atomicAdd(cursor + p, 1u)] = i;
  }
}

// Level 0: the seeds.
__global__ void __launch_bounds__(256) k_bfs_seeds(const int32_t* __restrict__ seed_list,
                                                   int32_t* __restrict__ frontier, DevStatus* st) {
  const int stride = gridDim.x * blockDim.x, ns = (int)st->n_seeds;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < ns; k += stride) frontier[k] = seed_list[k];
  if (blockIdx.x == 0 && threadIdx.x == 0) st->bfs_count[0] = (uint32_t)ns;
}

// One level: every frontier point hands its seed to its followers, which form the next frontier.
// off[p] .. off[p] + counts[p] is p's run (off = the scanned counts before the fill advanced
// them, i.e. the cursor minus the count).
__global__ void __launch_bounds__(256) k_bfs_level(const uint32_t* __restrict__ end, const uint32_t* __restrict__ counts,
                                                   const int32_t* __restrict__ followers, int32_t* __restrict__ par,
                                                   const int32_t* __restrict__ fin, int32_t* __restrict__ fout,
                                                   DevStatus* st, int level) {
  const uint32_t nin = st->bfs_count[level];
  if (nin == 0) return;
  const int stride = gridDim.x * blockDim.x;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < (int)nin; t += stride) {
    const int u = fin[t];
    const int seed = level == 0 ? u : par[u];
    const uint32_t e = end[u], b = e - counts[u];
    for (uint32_t q = b; q < e; ++q) {
      const int c = followers[q];
      par[c] = seed;
      if (counts[c]) fout[atomicAdd(&st->bfs_count[level + 1], 1u)] = c;  // leaves end the walk
    }
  }
}

int grid_for(int n, int threads) {
  int b = (n + threads - 1) / threads;
  const int cap = 148 * 32;
  return b < 1 ? 1 : (b > cap ? cap : b);
}

inline int chunk_grid(const KParams& kp) { return kp.n / kChunk + kp.ntiles + 1; }

inline Events events_of(Workspace& ws) { return Events{ws.ev, ws.ev_pt, ws.ev_tile, ws.ev_chunk}; }

template <int N, int MT>
void launch_density(const KParams& kp, Workspace& ws, cudaStream_t s) {
  k_density<N, MT><<<chunk_grid(kp), kTileThreads, 0, s>>>(kp, events_of(ws), ws.offsets, ws.chunk_tile,
                                                            ws.chunk_count, ws.chunk_total, ws.rec_w, ws.mq,
                                                            ws.rec_r);
}
template <int N, int MT>
void launch_nh(const KParams& kp, Workspace& ws, const clue_outputs& out, cudaStream_t s) {
  const SeedBufs sb{ws.par, kp.flags & CLUE_FLAG_NEAR_TIES ? ws.nh_s : nullptr, ws.seed_bits, ws.seed_list};
  // a block needed by at most this many lanes is split among all lanes
  const int split_lanes = std::max(0, std::min(16, (int)ws.tune_nh_split));
  if (kp.tiebreak == CLUE_TIE_RHO_INDEX)
    k_nearest_higher<N, MT, CLUE_TIE_RHO_INDEX><<<chunk_grid(kp), kTileThreads, 0, s>>>(
        kp, events_of(ws), ws.offsets, ws.chunk_tile, ws.chunk_count, ws.chunk_total, ws.rec_m_cur, ws.mq, ws.blk,
        ws.sblk, ws.perm, sb, out, ws.status, split_lanes);
  else
    k_nearest_higher<N, MT, CLUE_TIE_REFERENCE><<<chunk_grid(kp), kTileThreads, 0, s>>>(
        kp, events_of(ws), ws.offsets, ws.chunk_tile, ws.chunk_count, ws.chunk_total, ws.rec_m_cur, ws.mq, ws.blk,
        ws.sblk, ws.perm, sb, out, ws.status, split_lanes);
}
template <int N, int MT, int FORM>
void launch_density_spatial_form(const KParams& kp, Workspace& ws, cudaStream_t s, float kexp) {
  k_density_spatial<N, MT, FORM><<<chunk_grid(kp), kTileThreads, 0, s>>>(
      kp, events_of(ws), ws.offsets, ws.chunk_tile, ws.chunk_count, ws.chunk_total, ws.rec_m_cur, ws.mq,
      ws.blk, ws.sblk, ws.rec_r, kexp);
}
template <int N, int MT>
void launch_density_spatial(const KParams& kp, Workspace& ws, cudaStream_t s) {
  const float log2e = 1.4426950408889634f;
  if (kp.kernel_type == CLUE_KERNEL_EXPONENTIAL && kp.kpar[1] == 1.0f)
    launch_density_spatial_form<N, MT, kDensExpUnit>(kp, ws, s, -kp.kpar[0] * log2e);
  else if (kp.kernel_type == CLUE_KERNEL_GAUSSIAN && kp.kpar[0] == 0.0f && kp.kpar[2] == 1.0f)
    launch_density_spatial_form<N, MT, kDensGauss0Unit>(kp, ws, s, -kp.ginv * log2e);
  else
    launch_density_spatial_form<N, MT, kDensGeneric>(kp, ws, s, 0.0f);
}
// Symmetric density: kernel form and largest kernel value (the self term is 1).
template <int N, int MT, int FORM, int VAR>
void launch_density_sym_var(const KParams& kp, Workspace& ws, cudaStream_t s, float kexp, float kmax) {
  k_density_sym<N, MT, FORM, VAR><<<chunk_grid(kp), kTileThreads, 0, s>>>(
      kp, events_of(ws), ws.offsets, ws.chunk_tile, ws.chunk_count, ws.chunk_total, ws.rec_m_cur, ws.mq, ws.tblk_off,
      ws.tblk, ws.rec_r, ws.rho_fix, kexp, kmax, ws.status);
}
template <int N, int MT, int FORM>
void launch_density_sym_form(const KParams& kp, Workspace& ws, cudaStream_t s, float kexp, float kmax) {
  // the pair-step alternatives are built for the Euclidean metric and the unit-amplitude forms
  // in up to four dimensions (the benchmark configurations); elsewhere the plain step runs
  if constexpr (MT == CLUE_METRIC_EUCLIDEAN && FORM != kDensGeneric && N <= 4) {
    const int var = (ws.tune_density_gate ? 1 : 0) | (ws.tune_density_exp2 ? 2 : 0);
    switch (var) {
      case 1: launch_density_sym_var<N, MT, FORM, 1>(kp, ws, s, kexp, kmax); return;
      case 2: launch_density_sym_var<N, MT, FORM, 2>(kp, ws, s, kexp, kmax); return;
      case 3: launch_density_sym_var<N, MT, FORM, 3>(kp, ws, s, kexp, kmax); return;
      default: break;
    }
  }
  launch_density_sym_var<N, MT, FORM, 0>(kp, ws, s, kexp, kmax);
}
template <int N, int MT>
void launch_density_sym(const KParams& kp, Workspace& ws, cudaStream_t s, bool fuse_combine) {
  const float log2e = 1.4426950408889634f;
  float kmax = 1.0f;
  if (kp.kernel_type == CLUE_KERNEL_FLAT) kmax = fmaxf(1.0f, fabsf(kp.kpar[0]));
  if (kp.kernel_type == CLUE_KERNEL_EXPONENTIAL) kmax = fmaxf(1.0f, fabsf(kp.kpar[1]));
  if (kp.kernel_type == CLUE_KERNEL_GAUSSIAN) kmax = fmaxf(1.0f, fabsf(kp.kpar[2]));
  if (kp.kernel_type == CLUE_KERNEL_EXPONENTIAL && kp.kpar[1] == 1.0f)
    launch_density_sym_form<N, MT, kDensExpUnit>(kp, ws, s, -kp.kpar[0] * log2e, kmax);
  else if (kp.kernel_type == CLUE_KERNEL_GAUSSIAN && kp.kpar[0] == 0.0f && kp.kpar[2] == 1.0f)
    launch_density_sym_form<N, MT, kDensGauss0Unit>(kp, ws, s, -kp.ginv * log2e, kmax);
  else
    launch_density_sym_form<N, MT, kDensGeneric>(kp, ws, s, 0.0f, kmax);
  if (fuse_combine) {
    ws.sym_kmax = kmax;  // the combine runs with the nearest-higher block boxes
  } else {
    k_density_combine<N><<<grid_for(kp.n, 256), 256, 0, s>>>(kp, events_of(ws), kp.n, ws.rho_fix, ws.rec_r, kmax);
  }
}
// The symmetric sweep covers exactly the reference's candidates when the metric bounds every
// coordinate difference and no coordinate wraps.
inline bool symmetric_density_ok(const KParams& kp, int metric, int ndim) {
  if (metric != CLUE_METRIC_EUCLIDEAN && metric != CLUE_METRIC_MANHATTAN && metric != CLUE_METRIC_CHEBYSHEV)
    return false;
  for (int d = 0; d < ndim; ++d)
    if (kp.wrapped[d]) return false;
  return true;
}
template <int N>
void launch_density_sym_metric(int metric, const KParams& kp, Workspace& ws, cudaStream_t s, bool fuse_combine) {
  if (metric == CLUE_METRIC_MANHATTAN)
    launch_density_sym<N, CLUE_METRIC_MANHATTAN>(kp, ws, s, fuse_combine);
  else if (metric == CLUE_METRIC_CHEBYSHEV)
    launch_density_sym<N, CLUE_METRIC_CHEBYSHEV>(kp, ws, s, fuse_combine);
  else
    launch_density_sym<N, CLUE_METRIC_EUCLIDEAN>(kp, ws, s, fuse_combine);
}
template <int N, int MT>
void launch_near_ties(const KParams& kp, Workspace& ws, cudaStream_t s) {
  k_near_ties<N, MT><<<chunk_grid(kp), kTileThreads, 0, s>>>(
      kp, events_of(ws), ws.offsets, ws.chunk_tile, ws.chunk_count, ws.chunk_total, ws.rec_r, ws.rec_m_cur,
      ws.mq, ws.blk, ws.sblk, ws.nh_s, ws.status);
}

// Whether k_build takes the call: keys of 32 bits, and sizes where a few clusters beat the whole
// chip's separate launches.  Whole calls, k_build against separate launches: one flat 2-D event of 16k
// points 134 against 180 us, 40k 173 / 233, 65k 183 / 233, 131k 261 / 283 (a 3-D one with the symmetric
// density 293 / 304); 24 events of 3300 4-D points 167 / 246, 64 events 269 / 318, 100 2-D events of
// 3300 points 293 / 333, 300 events 798 / 756.
// Many events: a CTA of 512 threads takes one through all passes, however small, so the stage grows
// with the events beside the points.  2-D batches, exponential kernel: 1000 events of 10 points 203 against
// 259 us, 2500 361 / 354; 1500 of 100 points 269 / 277, 2500 385 / 349; 1500 of 250 points 356 / 358, 2000
// 435 / 423 (100000 events of 5 points: 11.5 against 6.5 ms).
// Many tiles: one CTA scans all tiles of an event and a batch's unused slots are launched, which the
// separate launches of the symmetric density (one sort) do not make up for beyond a line in points and
// tiles.  Single events: 16k points and 8192 tiles 203 / 223 us, 16384 tiles 261 / 249; 65k and 5461 202 /
// 210, 8192 238 / 228; 131k and 1024 203 / 201, 8192 287 / 249, 32768 592 / 396.  Batches: 8 events of 30000
// points and 1875 tiles each 323 / 336, 3750 461 / 441, 7500 713 / 613; 50 of 10000 points and 625 tiles 459 /
// 465, 1250 706 / 691, 2500 1105 / 1049; 24 of 3300 points and 1650 tiles 421 / 466.  The three sorts of the
// other calls take more with as many tiles (131k points and 65536 tiles, tile stage: 226 / 291 us).
constexpr int kBuildPoints = 131072;       // of a single event
constexpr int kBuildBatchPoints = 1 << 19;  // of a batch, each event at most kBuildEventPoints
constexpr int kBuildEventPoints = 32768;
constexpr int kBuildEvents = 2304;         // events + points / 512 of a batch
constexpr int kBuildTileBits = 16;
constexpr int kBuildSymTiles = 13000;      // symmetric density: tiles + points / 11 of a single event,
constexpr int kBuildSymEventTiles = 2048;  // tiles of a batch's event and
constexpr int kBuildSymBatchTiles = 49152;  // of a batch
inline bool build_takes(const KParams& kp, int max_points, int max_tiles, int tile_bits, int mbits, bool symmetric) {
  if (tile_bits > kBuildTileBits || tile_bits + mbits > 32) return false;
  if (kp.n_events == 1) return kp.n <= kBuildPoints && (!symmetric || kp.ntiles + kp.n / 11 <= kBuildSymTiles);
  if (kp.n_events + kp.n / 512 > kBuildEvents) return false;
  if (symmetric && (max_tiles > kBuildSymEventTiles || kp.ntiles > kBuildSymBatchTiles)) return false;
  // a batch's chunks and blocks have slots per event (k_build): they must fit the buffers
  return kp.n <= kBuildBatchPoints && max_points <= kBuildEventPoints && kp.n / 32 + kp.ntiles + 1 <= kp.n;
}
// CTAs per cluster: of 1024 threads for a single event, about a point per thread up to 16 CTAs (6k
// points: 8 CTAs 122 us, 16 123; 16k: 8 CTAs 136 us, 16 134; 65k: 209, 183); of 512 threads for a batch,
// as many as leave the clusters on the chip together (24 events: 8 CTAs 167 us, 4 176; 100 events: 4
// CTAs 293 us, 8 319, 2 317).  16 is beyond the portable cluster size, which the launch asks for.
inline int build_ranks(int n_events, int n) {
  if (n_events == 1) return n <= 1024 ? 1 : (n <= 2048 ? 2 : (n <= 4096 ? 4 : (n <= 8192 ? 8 : 16)));
  return n_events <= 64 ? 8 : (n_events <= 128 ? 4 : (n_events <= 256 ? 2 : 1));
}

#if CLUE_DEVICE_CHECKS
// The checked build can be told to find a device's limits: CLUE_BUILD_CLUSTERS = "fit N" (no clusters
// above N CTAs, 0: none), "refuse" (launches fail), "half", "double" (clusters of another size than
// asked for).
inline const char* build_clusters_env() {
  const char* v = getenv("CLUE_BUILD_CLUSTERS");
  return v ? v : "";
}
inline bool build_cluster_allowed(int ranks) {
  const char* v = build_clusters_env();
  return strncmp(v, "fit ", 4) != 0 || ranks <= atoi(v + 4);
}
inline cudaError_t build_launch_fault(cudaLaunchConfig_t& cfg, cudaLaunchAttribute& attr) {
  const char* v = build_clusters_env();
  if (!strcmp(v, "refuse")) return cudaErrorInvalidConfiguration;
  unsigned& c = attr.val.clusterDim.x;
  if (!strcmp(v, "half")) c = std::max(1u, c / 2);
  if (!strcmp(v, "double")) c = std::min(8u, c * 2);
  cfg.gridDim.x = (cfg.gridDim.x + c - 1) / c * c;
  return cudaSuccess;
}
#else
inline bool build_cluster_allowed(int) { return true; }
inline cudaError_t build_launch_fault(cudaLaunchConfig_t&, cudaLaunchAttribute&) { return cudaSuccess; }
#endif

// The launch of k_build with clusters of `ranks` CTAs.
template <int N, int W>
struct BuildLaunch {
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t cfg = {};
  BuildLaunch(int n_events, int ranks, cudaStream_t s) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)ranks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)(n_events * ranks));
    cfg.blockDim = dim3(32 * W);
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
  }
};

// Whether the current device can hold a cluster of `ranks` CTAs (a partitioned one may not); asked once
// per device and size.
template <int N, int W>
bool build_cluster_fits(int ranks) {
  constexpr int kDevices = 64;
  static std::atomic<uint32_t> known[kDevices];  // bit ranks: fits, bit 31 - ranks / 2: asked
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  const uint32_t fits = 1u << ranks, asked = 1u << (31 - ranks / 2);
  if (dev < kDevices) {
    const uint32_t k = known[dev].load(std::memory_order_relaxed);
    if (k & asked) return k & fits;
  }
  BuildLaunch<N, W> l(1, ranks, nullptr);
  int count = 0;
  cudaError_t e = cudaSuccess;
  if (ranks > 8) e = cudaFuncSetAttribute(k_build<N, W>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&count, k_build<N, W>, &l.cfg);
  if (e != cudaSuccess) cudaGetLastError();
  const bool ok = build_cluster_allowed(ranks) && e == cudaSuccess && count > 0;
  if (dev < kDevices) known[dev].fetch_or(asked | (ok ? fits : 0u), std::memory_order_relaxed);
  return ok;
}

template <int N, int W>
cudaError_t launch_build_cluster(const KParams& kp, const InPtrs& in, EvGrid* eg, const BuildBufs& o, bool two,
                                 int mbits, int tile_passes, int passes, int ranks, cudaStream_t s) {
  BuildLaunch<N, W> l(kp.n_events, ranks, s);
  cudaError_t e = build_launch_fault(l.cfg, l.attr[0]);
  if (e == cudaSuccess) e = cudaLaunchKernelEx(&l.cfg, k_build<N, W>, kp, in, eg, o, two, mbits, tile_passes, passes);
  if (e != cudaSuccess) cudaGetLastError();
  return e;
}

// Stage 1 through k_build with the largest clusters up to build_ranks that the device holds; returns
// the launches, 0 if there was none: the separate launches then take its place.
template <int N>
int launch_build(const KParams& kp, const InPtrs& in, Workspace& ws, bool two, int mbits, int tile_bits,
                 cudaStream_t s) {
  const int passes = (tile_bits + mbits + kRadixBits - 1) / kRadixBits;
  const int tile_passes = std::max(1, (tile_bits + kRadixBits - 1) / kRadixBits);
  const bool odd = passes & 1;
  const bool single = kp.n_events == 1;
  int ranks = build_ranks(kp.n_events, kp.n);
  while (ranks > 0 && !(single ? build_cluster_fits<N, 32>(ranks) : build_cluster_fits<N, 16>(ranks))) ranks /= 2;
  ws.build_ranks = ranks;
  if (ranks == 0) return 0;
  BuildBufs o{};
  o.k0 = ws.keys[0];
  o.k1 = ws.keys[1];
  o.k2 = ws.mkeys_alt;
  o.va = ws.vals[0];
  o.vb = ws.vals[1];
  o.perm = ws.mq_alt;
  o.vt = ws.nh_s;   // (nearest highers, label parents: not in use yet)
  o.inv = ws.par;
  o.rec_w = ws.rec_w;
  o.off = ws.offsets;
  o.chunk_off = ws.chunk_count;
  o.tblk_off = two ? nullptr : ws.tblk_off;
  o.chunk_tile = ws.chunk_tile;
  o.chunk_total = ws.chunk_total;
  o.tblk = two ? nullptr : ws.tblk;
  o.rho_fix = two ? nullptr : ws.rho_fix;
  o.seed_bits = ws.seed_bits;
  o.ev_pt = ws.ev_pt;
  o.ev_tile = ws.ev_tile;
  o.ev_chunk = ws.ev_chunk;
  o.st = ws.status;
  ws.perm = two ? ws.mq_alt : (odd ? ws.vals[0] : ws.vals[1]);
  ws.mq = two ? (odd ? ws.vals[1] : ws.vals[0]) : nullptr;
  if (!single)
    k_init<N><<<grid_for(std::max(kp.n_events, kp.n / 128), 256), 256, 0, s>>>(kp, events_of(ws), ws.ev_pt, ws.ev_tile,
                                                                               ws.seed_bits, ws.chunk_total, ws.status);
  const cudaError_t e =
      single ? launch_build_cluster<N, 32>(kp, in, ws.ev, o, two, mbits, tile_passes, passes, ranks, s)
             : launch_build_cluster<N, 16>(kp, in, ws.ev, o, two, mbits, tile_passes, passes, ranks, s);
  if (e != cudaSuccess) {
    ws.build_ranks = 0;
    return 0;
  }
  return single ? 1 : 2;
}

#define CLUE_METRIC_SWITCH(mt, FN, ...)                                           \
  switch (mt) {                                                                   \
    case CLUE_METRIC_EUCLIDEAN: FN<N, CLUE_METRIC_EUCLIDEAN>(__VA_ARGS__); break; \
    case CLUE_METRIC_WEIGHTED_EUCLIDEAN:                                          \
      FN<N, CLUE_METRIC_WEIGHTED_EUCLIDEAN>(__VA_ARGS__);                         \
      break;                                                                      \
    case CLUE_METRIC_PERIODIC_EUCLIDEAN:                                          \
      FN<N, CLUE_METRIC_PERIODIC_EUCLIDEAN>(__VA_ARGS__);                         \
      break;                                                                      \
    case CLUE_METRIC_MANHATTAN: FN<N, CLUE_METRIC_MANHATTAN>(__VA_ARGS__); break; \
    case CLUE_METRIC_CHEBYSHEV: FN<N, CLUE_METRIC_CHEBYSHEV>(__VA_ARGS__); break; \
    default: FN<N, CLUE_METRIC_WEIGHTED_CHEBYSHEV>(__VA_ARGS__); break;           \
  }

}  // namespace

// Pointer-jumping rounds of a run whose caller does not read the status back (rounds past the first
// do nothing unless the round before left a chain unresolved), and a round's passes.
constexpr int kJumpLaunches = 4;
constexpr JumpLimits kJumpLimits = {16, 256};
inline JumpLimits jump_limits() {
#if CLUE_DEVICE_CHECKS
  // (the checked build can be told to leave chains to later rounds)
  if (const char* v = getenv("CLUE_LABEL_HOPS")) return {std::max(1, atoi(v)), 1};
#endif
  return kJumpLimits;
}
// Blocks of the label climbs: no more than the GPU holds at once (see jump).
inline int label_blocks(int n) { return std::min(grid_for(n, 256), 148 * 8); }

template <int N>
clue_status run_pipeline(Workspace& ws, const RunArgs& a, cudaStream_t s) {
  KParams kp = a.kp;
  kp.one = 1.0f;
  const int n = kp.n;
  InPtrs in{};
  for (int d = 0; d < N; ++d) in.c[d] = a.coords[d];
  in.w = a.weight;
  const Events ev = events_of(ws);
  ws.near_from_host = false;  // this run's counts land in the device status block

  stage_mark(ws, 0, s);
  int launches = 0;
  // density order: the reference's candidate order for the flat kernel (bit-exact sums), spatial
  // order for the exponential and Gaussian kernels (whose device expf already differs from the
  // host's by an ulp) unless the caller asks for the reference order
  const bool spatial_density = (kp.flags & CLUE_FLAG_REFERENCE_ORDER) == 0 &&
                               (kp.kernel_type != CLUE_KERNEL_FLAT || (kp.flags & CLUE_FLAG_SPATIAL_DENSITY) != 0);
  const bool symmetric =
      spatial_density && symmetric_density_ok(kp, a.metric, N) && ws.tblk && ws.tblk_off && ws.rho_fix &&
      ws.tune_symmetric != 0;
  const int bits = bits_for((uint32_t)(kp.ntiles - 1));
  const int mbits = MortonSortBits<N>::kBits;
  const int nsb = (n + 1023) >> 10;
  const int max_slots = kChunkWarps * (n / kChunk + kp.ntiles + 1);
  const int pts_max = kp.n_events == 1 ? n : a.max_points;
  const int tiles_max = kp.n_events == 1 ? kp.ntiles : a.max_tiles;
  const int ev_bits = bits_for((uint32_t)(tiles_max - 1));
  bool composite = symmetric;
  ws.build_ranks = 0;
  int built = 0;
  if (build_takes(kp, pts_max, tiles_max, ev_bits, mbits, symmetric))
    built = launch_build<N>(kp, in, ws, !symmetric, mbits, ev_bits, s);
  launches += built;
  if (built == 0) {
    launches += 4;  // init, bbox, grid, bin
    k_init<N><<<grid_for(std::max(kp.n_events, n / 128), 256), 256, 0, s>>>(kp, ev, ws.ev_pt, ws.ev_tile, ws.seed_bits,
                                                                            nullptr, ws.status);
    if (symmetric) cudaMemsetAsync(ws.rho_fix, 0, (size_t)n * sizeof(int64_t), s);
    if (kp.n_events == 1) {
      k_bbox_single<N><<<std::max(1, std::min(grid_for(n, 1024), 148 * 4)), 256, 0, s>>>(in, n, ws.ev, ws.status);
    } else {
      // spans of 32..1024 points: about four spans per resident warp (64 per SM) when there
      // are enough points, so the loads of many spans are in flight
      const int span = std::max(32, std::min(1024, (n / (148 * 64 * 4)) & ~31));
      const int blocks = std::max(1, std::min(grid_for(n, 256), ((n + span - 1) / span + 7) / 8));
      if (ws.ev_chunk) {
        k_event_chunks<<<grid_for(kp.n_events, 256), 256, 0, s>>>(kp.n_events, ws.ev_pt, ws.ev_chunk);
        ++launches;
      }
      k_bbox_events<N><<<blocks, 256, 0, s>>>(in, n, kp.n_events, ws.ev_pt, ws.ev_chunk, ws.ev, ws.status, span);
    }
    k_grid<N><<<grid_for(kp.n_events, 256), 256, 0, s>>>(kp.n_events, ws.ev);
    // The symmetric sweep needs no tile order by point index: one sort by (tile, Morton) composite
    // keys gives its record order, and positions inside a tile are only compared through the
    // points' indices.  The other sweeps take the tile order by index and a Morton order beside it.
    composite = symmetric && bits + mbits <= 32;
    if (composite) {
      k_bin_composite<N><<<grid_for(n, 1024), 256, 0, s>>>(kp, in, ev, mbits, ws.keys[0]);
      const int cur = radix_sort_pairs(ws.keys, ws.vals, true, n, bits + mbits, ws.hist, ws.scan_scratch, s);
      ws.perm = ws.vals[cur];
      offsets_from_sorted(ws.keys[cur], n, kp.ntiles, ws.offsets, s, mbits);
      ws.mq = nullptr;
      k_gather<N><<<grid_for(n, 256), 256, 0, s>>>(in, n, ws.perm, ws.rec_w, ws.status);
      launches += radix_sort_launches(bits + mbits) + 2;
    } else {
      k_bin<N><<<grid_for(n, 256), 256, 0, s>>>(kp, in, ev, ws.keys[0]);
      const int cur = radix_sort_pairs(ws.keys, ws.vals, true, n, bits, ws.hist, ws.scan_scratch, s);
      ws.perm = ws.vals[cur];
      const uint32_t* sorted_keys = ws.keys[cur];
      offsets_from_sorted(sorted_keys, n, kp.ntiles, ws.offsets, s);
      k_gather<N><<<grid_for(n, 256), 256, 0, s>>>(in, n, ws.perm, ws.rec_w, ws.status);
      // fine Morton order inside every tile: a stable sort by Morton key, then a stable sort by
      // tile; mq[p] = tile-sorted position of the p-th record in (tile, Morton) order
      uint32_t* mkeys[2] = {ws.keys[cur ^ 1], ws.mkeys_alt};
      int32_t* mvals[2] = {ws.vals[cur ^ 1], ws.mq_alt};
      k_morton_keys<N><<<grid_for(n, 256), 256, 0, s>>>(kp, ev, ws.rec_w, sorted_keys, mkeys[0]);
      int mc = radix_sort_pairs(mkeys, mvals, true, n, MortonSortBits<N>::kBits, ws.hist, ws.scan_scratch, s);
      if (mc != 0) {
        std::swap(mkeys[0], mkeys[1]);
        std::swap(mvals[0], mvals[1]);
      }
      k_tile_of<<<grid_for(n, 256), 256, 0, s>>>(sorted_keys, mvals[0], n, mkeys[0]);
      mc = radix_sort_pairs(mkeys, mvals, false, n, bits, ws.hist, ws.scan_scratch, s);
      ws.mq = mvals[mc];
      launches += 2 * radix_sort_launches(bits) + 2 + 1 + radix_sort_launches(MortonSortBits<N>::kBits) + 1;
    }
    k_tile_counts<<<grid_for(kp.ntiles, 256), 256, 0, s>>>(kp.ntiles, ws.offsets, ws.chunk_count,
                                                           symmetric ? ws.tblk_off : nullptr);
    exclusive_scan(ws.chunk_count, ws.chunk_count, (size_t)kp.ntiles, ws.scan_scratch, ws.chunk_total, s);
    if (symmetric) exclusive_scan(ws.tblk_off, ws.tblk_off, (size_t)kp.ntiles, ws.scan_scratch, nullptr, s);
    k_chunk_map<<<grid_for(kp.ntiles, 256), 256, 0, s>>>(kp.ntiles, ws.offsets, ws.chunk_count, ws.chunk_tile);
    launches += 1 + scan_launches(kp.ntiles) * (symmetric ? 2 : 1) + 1;
    if (symmetric) {
      if (!composite) {
        k_gather_morton<N><<<grid_for(n, 256), 256, 0, s>>>(ws.rec_w, n, ws.mq, ws.rec_m);
        ++launches;
      }
      k_tblock_bbox<N><<<grid_for(max_slots, 256), 256, 0, s>>>(max_slots, ws.chunk_total, ws.offsets, ws.chunk_tile,
                                                                 ws.chunk_count, ws.tblk_off,
                                                                 composite ? ws.rec_w : ws.rec_m, ws.tblk);
      ++launches;
    }
  }
  ws.rec_m_cur = composite ? ws.rec_w : ws.rec_m;
  if (spatial_density && !symmetric) {
    k_boxes<N, true><<<nsb, 1024, 0, s>>>(kp, ev, ws.mq, ws.rec_w, ws.rec_m, nullptr, 0.0f, ws.blk, ws.sblk);
    ++launches;
  }

  stage_mark(ws, 1, s);
  if (symmetric) {
    launch_density_sym_metric<N>(a.metric, kp, ws, s, composite);
  } else if (spatial_density) {
    CLUE_METRIC_SWITCH(a.metric, launch_density_spatial, kp, ws, s);
  } else {
    CLUE_METRIC_SWITCH(a.metric, launch_density, kp, ws, s);
  }
  launches += symmetric && !composite ? 2 : 1;  // (a composite run combines with the block boxes)
  stage_mark(ws, 2, s);
  // Morton-ordered copy of the records with their densities (the tile-ordered records themselves
  // after a composite sort, where the density's fixed-point sums are added in here) and its block
  // and super-block boxes with the largest rho, for the nearest-higher search
  if (composite) {
    k_boxes<N, false><<<nsb, 1024, 0, s>>>(kp, ev, nullptr, ws.rec_r, nullptr, ws.rho_fix, ws.sym_kmax, ws.blk, ws.sblk);
    ws.rec_m_cur = ws.rec_r;
  } else {
    k_boxes<N, true><<<nsb, 1024, 0, s>>>(kp, ev, ws.mq, ws.rec_r, ws.rec_m, nullptr, 0.0f, ws.blk, ws.sblk);
    ws.rec_m_cur = ws.rec_m;
  }
  CLUE_METRIC_SWITCH(a.metric, launch_nh, kp, ws, a.out, s);
  if (kp.flags & CLUE_FLAG_NEAR_TIES) {
    CLUE_METRIC_SWITCH(a.metric, launch_near_ties, kp, ws, s);
    ++launches;
  }
  stage_mark(ws, 3, s);
  const size_t words = ((size_t)n + 31) / 32;
  if (words <= kScanOneBlock) {
    const int blocks = std::min(kSeedBlocks, (n + kSeedBlockPoints - 1) / kSeedBlockPoints);
    k_seed_labels_scan<<<blocks, 1024, 0, s>>>(kp, ev, ws.seed_bits, ws.seed_total, (int)words, ws.seed_list, ws.perm,
                                               ws.par, a.ev_n_seeds, a.ev_n_clusters, ws.status);
    launches += 1;
  } else {
    exclusive_scan_bits(ws.seed_bits, ws.seed_rank, words, ws.scan_scratch, ws.seed_total, s);
    k_seed_labels<<<std::min(grid_for(std::max(kp.n_events, n / 8), 256), 148 * 8), 256, 0, s>>>(
        kp, ev, ws.seed_bits, ws.seed_rank, ws.seed_total, ws.seed_list, ws.perm, ws.par, a.ev_n_seeds,
        a.ev_n_clusters, ws.status);
    launches += scan_launches(words) + 1;
  }
  if (ws.tune_labels_bfs) {
    // follower CSR in buffers that are dead by now: the sort keys and the weight records
    uint32_t* counts = ws.keys[0];
    uint32_t* run_end = ws.keys[1];
    int32_t* followers = reinterpret_cast<int32_t*>(ws.rec_w);
    int32_t* front[2] = {followers + n, followers + 2 * (size_t)n};
    cudaMemsetAsync(counts, 0, (size_t)n * sizeof(uint32_t), s);
    k_follower_count<<<grid_for(n, 256), 256, 0, s>>>(ws.par, n, counts);
    exclusive_scan(counts, run_end, (size_t)n, ws.scan_scratch, nullptr, s);
    k_follower_fill<<<grid_for(n, 256), 256, 0, s>>>(ws.par, n, run_end, followers);
    k_bfs_seeds<<<std::min(grid_for(n, 256), 148 * 8), 256, 0, s>>>(ws.seed_list, front[0], ws.status);
    const int lg = std::min(grid_for(n, 256), 148 * 8);
    for (int l = 0; l < kBfsLevels; ++l)
      k_bfs_level<<<lg, 256, 0, s>>>(run_end, counts, followers, ws.par, front[l & 1], front[(l + 1) & 1], ws.status,
                                     l);
    launches += scan_launches(n) + kBfsLevels + 3;  // count, scan, fill, seeds, levels
  }
  (n < kLabelChainPoints ? k_labels<1> : k_labels<4>)<<<label_blocks(n), 256, 0, s>>>(
      ws.par, ws.perm, a.out.cluster_index, n, jump_limits(), a.blocking ? 1 : kJumpLaunches, ws.status);
  if (!a.blocking) {
    for (int r = 1; r < kJumpLaunches; ++r)
      k_jump<<<label_blocks(n), 256, 0, s>>>(ws.par, n, jump_limits(), ws.status, r);
    k_labels_again<<<grid_for(n, 256), 256, 0, s>>>(ws.par, ws.perm, a.out.cluster_index, n, kJumpLaunches, ws.status);
  }
  stage_mark(ws, 4, s);
  // Morton boxes, nearest higher, labels
  ws.launches += launches + 2 + (a.blocking ? 1 : 1 + kJumpLaunches);
  CLUE_CUDA_TRY(cudaGetLastError());
  return CLUE_OK;
}

// Continue pointer jumping from the host after the enqueued launches left chains
// unresolved (only for very deep nearest-higher chains); synchronises per launch.
template <int N>
clue_status finish_labels(Workspace& ws, const RunArgs& a, cudaStream_t s, int first_round) {
  const int n = a.kp.n;
  int r = first_round;
  for (uint32_t unres = 1; unres != 0 && r < 64; ++r) {
    k_jump<<<label_blocks(n), 256, 0, s>>>(ws.par, n, jump_limits(), ws.status, r);
    ++ws.launches;
    CLUE_CUDA_TRY(cudaMemcpyAsync(&unres, &ws.status->unresolved[r], 4, cudaMemcpyDeviceToHost, s));
    CLUE_CUDA_TRY(cudaStreamSynchronize(s));
  }
  k_labels_again<<<grid_for(n, 256), 256, 0, s>>>(ws.par, ws.perm, a.out.cluster_index, n, r, ws.status);
  ++ws.launches;
  CLUE_CUDA_TRY(cudaGetLastError());
  return CLUE_OK;
}

template clue_status run_pipeline<CLUE_NDIM>(Workspace&, const RunArgs&, cudaStream_t);
template clue_status finish_labels<CLUE_NDIM>(Workspace&, const RunArgs&, cudaStream_t, int);

}  // namespace clue_b200
