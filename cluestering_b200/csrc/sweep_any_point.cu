// sweep_any_point.cu — local density (core/detail/ClusteringKernels.hpp:29-140) and
// nearest higher (:142-291) off the fast path, with a warp per point: runs of at most
// 16,384 points (any_form).
//
// The lanes find the tiles of the point's search box, 32 at a time in the reference's
// order, and test their points 32 at a time in that order. For the density the lanes
// with a contribution put it, in order, in shared memory, and the sum is taken from
// there 64 at a time: it is a chain of rounded additions in the reference's order, but
// the distances and kernel values are not part of the chain. For the nearest higher
// every lane keeps its best, and the best of the lanes is the answer: the comparisons
// are a strict order on (distance, density, tag, visiting order).
// Bound by latency and, from about 16,384 points on, by instruction issue: a point
// loads its candidates for itself, where sweep_any.cu's block loads them once for 32.
// Density + nearest higher, us, a block per 32 points / a warp per point: 1,024 points
// with the periodic metric 24 + 28 / 13 + 14; 4,096 in 1-D 102 + 55 / 39 + 31; 16,384 in
// 4-D 112 + 116 / 95 + 101; but 32,768 with the periodic metric 171 + 136 / 232 + 234 and
// 131,072 1,594 + 821 / 2,413 + 2,328.
#include <cfloat>

#include "engine.h"
#include "sweep_device.cuh"

namespace clue_impl {

namespace {

constexpr int kWarps = kThreads / 32;
constexpr int kAhead = 2;       // rounds of candidates loaded together
constexpr int kSum = 64;        // contributions added together

// The last k in [0, 32) with start[k] <= x (start ascending, start[0] <= x).
__device__ __forceinline__ int last_at_or_before(const int* start, int x) {
  int k = 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    k += start[k + o] <= x ? o : 0;
  return k;
}

// The warp's point and its search box.
template <int D>
struct Point {
  int s;
  EventDesc ev;
  float x[D], sig[D];
  int inf[D], n[D];
  int64_t box;  // tiles of the box

  __device__ Point(const RunParams& p, const SweepArgs& a, int64_t w, float radius) : s((int)w) {
    ev = a.events[a.sevt[s]];
    const GridDesc& g = a.grids[ev.grid];
    load_point<D>(p, a, s, x, sig);
    int sup[D];
    search_box<D>(g, p, x, sig, radius, inf, sup);
    box = 1;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      n[d] = max(sup[d] - inf[d] + 1, 1);  // (a box whose ends cross is walked as one bin)
      box *= n[d];
    }
  }

  // The box's tile number k in visiting order (last dimension fastest): its first
  // sorted position and its number of points.
  __device__ void tile(const RunParams& p, const SweepArgs& a, int64_t k, int* begin, int* points) const {
    const GridDesc& g = a.grids[ev.grid];
    int b[D];
#pragma unroll
    for (int d = D - 1; d > 0; --d) {
      // (boxes of fewer than 2^31 tiles in all but the widest wrapped cases)
      const int64_t q = box <= INT32_MAX ? (int64_t)((int)k / n[d]) : k / n[d];
      b[d] = inf[d] + (int)(k - q * n[d]);
      k = q;
    }
    b[0] = inf[0] + (int)k;
    const int t = tile_id<D>(g, p, ev.tile_base, b);
    *begin = a.tile_offset[t];
    *points = a.tile_offset[t + 1] - *begin;
  }
};

// Calls body(q[kAhead], order, total) for the box's points in visiting order, kAhead
// rounds of 32 at a time: lane l's candidate of round u has sorted position q[u] (-1:
// none) and visiting number order + u * 32 + l. off and first are the warp's tables.
template <int D, typename Body>
__device__ __forceinline__ void for_each_round(const RunParams& p, const SweepArgs& a, const Point<D>& pt, int* off,
                                               int* first, Body&& body) {
  const int lane = threadIdx.x & 31;
  int order = 0;
  for (int64_t tb = 0; tb < pt.box; tb += 32) {
    int begin = 0, m = 0;
    if (tb + lane < pt.box)
      pt.tile(p, a, tb + lane, &begin, &m);
    int incl = m;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(kFullMask, incl, o);
      if (lane >= o)
        incl += y;
    }
    const int total = __shfl_sync(kFullMask, incl, 31);
    __syncwarp();
    off[lane] = incl - m;
    first[lane] = begin - (incl - m);
    __syncwarp();
    for (int c = 0; c < total; c += 32 * kAhead) {
      int q[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const int pos = c + u * 32 + lane;
        q[u] = pos < total ? first[last_at_or_before(off, pos)] + pos : -1;
      }
      body(q, order + c);
    }
    order += total;
  }
}

template <int D, int METRIC>
__global__ void __launch_bounds__(kThreads) k_density_point(const RunParams p, const SweepArgs a) {
  __shared__ int s_off[kWarps][32], s_first[kWarps][32];
  __shared__ __align__(16) float s_add[kWarps][kSum + 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t n = a.n;
  float* add = s_add[warp];
  // A candidate out of range adds 0 * k * w: +-0, which leaves a sum as it is,
  // unless k or w is infinite or NaN. Such candidates are evaluated like those in
  // range.
  const float den = __fmul_rn(__fmul_rn(2.0f, p.kernel_p0), p.kernel_p0);
  const bool all_special = !isfinite(p.kernel_p0) || !isfinite(p.kernel_p1) ||
                           (p.kernel_kind == CLUE_KERNEL_GAUSSIAN && !isfinite(den));
  const bool mahalanobis = METRIC == kAnyMetric && p.metric_kind == CLUE_METRIC_MAHALANOBIS;
  const float thr = metric_has_sqrt(p.metric_kind) ? p.dc2 : p.dc;
  for (int64_t w = (int64_t)blockIdx.x * kWarps + warp; w < n; w += (int64_t)gridDim.x * kWarps) {
    const Point<D> pt(p, a, w, p.dc);
    float rho = 0.0f;
    int held = 0;  // contributions in `add`
    for_each_round<D>(p, a, pt, s_off[warp], s_first[warp], [&](const int* q, int) {
      float xj[kAhead][D], sj[kAhead][D], wj[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        wj[u] = 0.0f;
        if (q[u] >= 0) {
#pragma unroll
          for (int d = 0; d < D; ++d) {
            xj[u][d] = a.sx[d * n + q[u]];
            sj[u][d] = mahalanobis ? a.ssig[d * n + q[u]] : 0.0f;
          }
          wj[u] = a.sw[q[u]];
        }
      }
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const float inner = inner_distance<D, METRIC>(p, pt.x, xj[u], pt.sig, sj[u]);
        const bool hit = q[u] >= 0 && (!(inner > thr) || all_special || !isfinite(wj[u]));
        const unsigned hits = __ballot_sync(kFullMask, hit);
        if (hits == 0)
          continue;
        if (hit) {
          const float dist = metric_finish(p, inner);
          const float kv = kernel_value(p, dist, q[u] == pt.s);
          // rho_i += static_cast<int>(distance <= density_radius) * k * w_j
          add[held + __popc(hits & ((1u << lane) - 1u))] =
              __fmul_rn(__fmul_rn((float)(int)(dist <= p.dc), kv), wj[u]);
        }
        held += __popc(hits);
        __syncwarp();
        if (held >= kSum) {
#pragma unroll
          for (int k = 0; k < kSum; k += 4) {
            const float4 v = *reinterpret_cast<const float4*>(add + k);
            rho = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(rho, v.x), v.y), v.z), v.w);
          }
          held -= kSum;
          const float rest = add[kSum + lane];  // at most 32 are left
          __syncwarp();
          add[lane] = rest;
          __syncwarp();
        }
      }
    });
    for (int k = 0; k < held; ++k)
      rho = __fadd_rn(rho, add[k]);
    __syncwarp();
    if (lane == 0) {
      a.srho[pt.s] = rho;
      if (a.out_rho)
        a.out_rho[a.perm[pt.s]] = rho;
    }
  }
}

struct AnyBest {
  float dist, hi;  // no candidate with metric_inner above hi can win
  int q, order;
  uint64_t key;
};

template <int D, int METRIC>
__global__ void __launch_bounds__(kThreads) k_nearest_higher_point(const RunParams p, const SweepArgs a) {
  __shared__ int s_off[kWarps][32], s_first[kWarps][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t n = a.n;
  const bool root = metric_has_sqrt(p.metric_kind);
  const bool mahalanobis = METRIC == kAnyMetric && p.metric_kind == CLUE_METRIC_MAHALANOBIS;
  for (int64_t w = (int64_t)blockIdx.x * kWarps + warp; w < n; w += (int64_t)gridDim.x * kWarps) {
    const Point<D> pt(p, a, w, p.dm);
    const int gi = a.perm[pt.s];
    const float rho_i = a.srho[pt.s];
    const float unc = p.has_unc ? a.sunc[pt.s] : 1.0f;
    const float min_density = __fmul_rn(p.rhoc, unc);
    const bool seedlike = rho_i >= min_density;
    // ClusteringKernels.hpp:168; as a bound on metric_inner
    const float eff = seedlike ? p.seed_dc : p.dm;
    const float eff_inner = root ? (seedlike ? p.seed2 : p.dm2) : eff;
    // ClusteringKernels.hpp:180-182 as one order on (density, tag): see rho_key;
    // equal densities count only above zero, else the tag part is saturated
    const bool nan_i = rho_i != rho_i;
    const uint32_t tag_i = p.has_tags ? a.stag[pt.s] : (uint32_t)gi;
    const uint64_t key_i = ((uint64_t)(nan_i ? 0xffffffffu : rho_key(rho_i)) << 32) |
                           ((nan_i || !(rho_i > 0.0f)) ? 0xffffffffu : tag_i);
    // no candidate at FLT_MAX or beyond is taken (the reference starts from there)
    AnyBest best{FLT_MAX, INFINITY, -1, 0, ~0ull};
    const auto wins = [&](float dist, uint64_t key, int order) {  // ClusteringKernels.hpp:195-202
      return (dist < best.dist) ||
             ((dist == best.dist) && ((key > best.key) || (key == best.key && order < best.order)));
    };
    for_each_round<D>(p, a, pt, s_off[warp], s_first[warp], [&](const int* q, int order) {
      float xj[kAhead][D], sj[kAhead][D];
      uint64_t key[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        key[u] = 0;
        if (q[u] >= 0) {
#pragma unroll
          for (int d = 0; d < D; ++d) {
            xj[u][d] = a.sx[d * n + q[u]];
            sj[u][d] = mahalanobis ? a.ssig[d * n + q[u]] : 0.0f;
          }
          key[u] = ((uint64_t)rho_key(a.srho[q[u]]) << 32) | (p.has_tags ? a.stag[q[u]] : (uint32_t)a.perm[q[u]]);
        }
      }
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        if (q[u] < 0 || key[u] <= key_i)
          continue;
        const float inner = inner_distance<D, METRIC>(p, pt.x, xj[u], pt.sig, sj[u]);
        if (inner <= eff_inner && inner <= best.hi) {
          const float dist = metric_finish(p, inner);
          if (dist <= eff && wins(dist, key[u], order + u * 32 + lane))
            // a larger root needs a square larger by 2^-23 relative; tiny squares stay open
            best = AnyBest{dist,
                           !root ? inner : inner >= 0x1p-100f ? __fmul_rn(inner, 1.00000095367431640625f) : INFINITY,
                           q[u], order + u * 32 + lane, key[u]};
        }
      }
    });
    __syncwarp();
    // the best of the lanes
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float dist = __shfl_xor_sync(kFullMask, best.dist, o);
      const int q = __shfl_xor_sync(kFullMask, best.q, o), order = __shfl_xor_sync(kFullMask, best.order, o);
      const uint64_t key = __shfl_xor_sync(kFullMask, best.key, o);
      if (q >= 0 && wins(dist, key, order))
        best = AnyBest{dist, 0.0f, q, order, key};
    }
    if (lane == 0) {
      const int nh = best.q >= 0 ? a.perm[best.q] : -1;
      a.out_nh[gi] = nh;
      a.parent[pt.s] = best.q >= 0 ? best.q : pt.s;
      // KernelFindClusters, ClusteringKernels.hpp:301-313
      const int seed = (nh == -1) && seedlike;
      a.seed_flag[gi] = seed;
      if (a.out_seed)
        a.out_seed[gi] = seed;
    }
  }
}

template <int D, int METRIC>
cudaError_t launch_point(bool density, const RunParams& p, const SweepArgs& a, cudaStream_t st) {
  const int blocks = (int)std::min<int64_t>((a.n + kWarps - 1) / kWarps, (int64_t)sm_count() * 256);
  if (density)
    k_density_point<D, METRIC><<<blocks, kThreads, 0, st>>>(p, a);
  else
    k_nearest_higher_point<D, METRIC><<<blocks, kThreads, 0, st>>>(p, a);
  count_launches(1);
  return cudaGetLastError();
}

template <int D>
cudaError_t launch_dim(bool density, const RunParams& p, const SweepArgs& a, cudaStream_t st) {
  switch (p.metric_kind) {
    case CLUE_METRIC_EUCLIDEAN: return launch_point<D, CLUE_METRIC_EUCLIDEAN>(density, p, a, st);
    case CLUE_METRIC_PERIODIC_EUCLIDEAN: return launch_point<D, CLUE_METRIC_PERIODIC_EUCLIDEAN>(density, p, a, st);
    default: return launch_point<D, kAnyMetric>(density, p, a, st);
  }
}

}  // namespace

cudaError_t launch_sweep_point(bool density, int D, const RunParams& p, const SweepArgs& a, cudaStream_t st) {
  switch (D) {
    case 1: return launch_dim<1>(density, p, a, st);
    case 2: return launch_dim<2>(density, p, a, st);
    case 3: return launch_dim<3>(density, p, a, st);
    case 4: return launch_dim<4>(density, p, a, st);
    case 5: return launch_dim<5>(density, p, a, st);
    case 6: return launch_dim<6>(density, p, a, st);
    case 7: return launch_dim<7>(density, p, a, st);
    case 8: return launch_dim<8>(density, p, a, st);
    case 9: return launch_dim<9>(density, p, a, st);
    case 10: return launch_dim<10>(density, p, a, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace clue_impl
