// sweep_any_thread.cu — local density (core/detail/ClusteringKernels.hpp:29-140) and
// nearest higher (:142-291) off the fast path, with a thread per point that walks its
// search box in the reference's order.
//
// The forms of sweep_any.cu and sweep_any_point.cu shorten a point's chain of loads,
// which bounds this one, and pay for it with work that every point or tile costs them.
// Where there are points enough to hide the chains, or few candidates to a point, this
// one is the fastest: any_form has the lines and the figures.
#include <cfloat>

#include "engine.h"
#include "sweep_device.cuh"

namespace clue_impl {

namespace {

template <int D>
__global__ void __launch_bounds__(kThreads) k_density_thread(const RunParams p, const SweepArgs a, const RunWhen when) {
  if (!runs_when(a, when))
    return;
  const int64_t n = a.n;
  const bool mahalanobis = p.metric_kind == CLUE_METRIC_MAHALANOBIS;
  for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < n; w += (int64_t)gridDim.x * blockDim.x) {
    const int s = a.work_dens ? a.work_dens[w] : (int)w;
    const EventDesc ev = a.events[a.sevt[s]];
    const GridDesc& g = a.grids[ev.grid];
    float xi[D], si[D];
    load_point<D>(p, a, s, xi, si);
    int inf[D], sup[D], b[D];
    search_box<D>(g, p, xi, si, p.dc, inf, sup);
#pragma unroll
    for (int d = 0; d < D; ++d)
      b[d] = inf[d];
    float rho = 0.0f;
    do {
      const int t = tile_id<D>(g, p, ev.tile_base, b);
      const int q1 = a.tile_offset[t + 1];
      for (int q = a.tile_offset[t]; q < q1; ++q) {
        float xj[D], sj[D];
#pragma unroll
        for (int d = 0; d < D; ++d) {
          xj[d] = a.sx[d * n + q];
          sj[d] = mahalanobis ? a.ssig[d * n + q] : 0.0f;
        }
        const float dist = metric_finish(p, metric_inner<D>(p, xi, xj, si, sj));
        const float k = kernel_value(p, dist, q == s);
        // rho_i += static_cast<int>(distance <= density_radius) * k * w_j
        rho = __fadd_rn(rho, __fmul_rn(__fmul_rn((float)(int)(dist <= p.dc), k), a.sw[q]));
      }
    } while (next_tile<D>(b, inf, sup));
    a.srho[s] = rho;
    if (a.out_rho)
      a.out_rho[a.perm[s]] = rho;
  }
}

template <int D>
__global__ void __launch_bounds__(kThreads)
    k_nearest_higher_thread(const RunParams p, const SweepArgs a, const RunWhen when) {
  if (!runs_when(a, when))
    return;
  const int64_t n = a.n;
  const bool mahalanobis = p.metric_kind == CLUE_METRIC_MAHALANOBIS;
  for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < n; w += (int64_t)gridDim.x * blockDim.x) {
    const int s = a.work_nh ? a.work_nh[w] : (int)w;
    const EventDesc ev = a.events[a.sevt[s]];
    const GridDesc& g = a.grids[ev.grid];
    float xi[D], si[D];
    load_point<D>(p, a, s, xi, si);
    const int gi = a.perm[s];
    const float rho_i = a.srho[s];
    const float unc = p.has_unc ? a.sunc[s] : 1.0f;
    const float min_density = __fmul_rn(p.rhoc, unc);
    // ClusteringKernels.hpp:168
    const float eff = (rho_i >= min_density) ? p.seed_dc : p.dm;
    const uint32_t tag_i = p.has_tags ? a.stag[s] : (uint32_t)gi;
    int inf[D], sup[D], b[D];
    search_box<D>(g, p, xi, si, p.dm, inf, sup);
#pragma unroll
    for (int d = 0; d < D; ++d)
      b[d] = inf[d];
    float delta = FLT_MAX;
    int nh = -1, nh_pos = s;
    float rho_nh = 0.0f;
    uint32_t tag_nh = 0;
    do {
      const int t = tile_id<D>(g, p, ev.tile_base, b);
      const int q1 = a.tile_offset[t + 1];
      for (int q = a.tile_offset[t]; q < q1; ++q) {
        const float rho_j = a.srho[q];
        const int gj = a.perm[q];
        const uint32_t tag_j = p.has_tags ? a.stag[q] : (uint32_t)gj;
        // ClusteringKernels.hpp:180-182
        const bool higher = (rho_j > rho_i) || ((rho_j == rho_i) && (rho_j > 0.0f) && (tag_j > tag_i));
        if (!higher)
          continue;
        float xj[D], sj[D];
#pragma unroll
        for (int d = 0; d < D; ++d) {
          xj[d] = a.sx[d * n + q];
          sj[d] = mahalanobis ? a.ssig[d * n + q] : 0.0f;
        }
        const float dist = metric_finish(p, metric_inner<D>(p, xi, xj, si, sj));
        // ClusteringKernels.hpp:195-202
        if (dist <= eff && ((dist < delta) || ((dist == delta) && (nh >= 0) &&
                                               ((rho_j > rho_nh) || ((rho_j == rho_nh) && (tag_j > tag_nh)))))) {
          delta = dist;
          nh = gj;
          nh_pos = q;
          rho_nh = rho_j;
          tag_nh = tag_j;
        }
      }
    } while (next_tile<D>(b, inf, sup));
    a.out_nh[gi] = nh;
    a.parent[s] = nh_pos;
    // KernelFindClusters, ClusteringKernels.hpp:301-313
    const int seed = (nh == -1) && (rho_i >= min_density);
    a.seed_flag[gi] = seed;
    if (a.out_seed)
      a.out_seed[gi] = seed;
  }
}

template <int D>
cudaError_t launch_dim(bool density, const RunParams& p, const SweepArgs& a, RunWhen when, cudaStream_t st) {
  const int blocks = (int)std::min<int64_t>((a.n + kThreads - 1) / kThreads, (int64_t)sm_count() * 16);
  if (density)
    k_density_thread<D><<<blocks, kThreads, 0, st>>>(p, a, when);
  else
    k_nearest_higher_thread<D><<<blocks, kThreads, 0, st>>>(p, a, when);
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_sweep_thread(bool density, int D, const RunParams& p, const SweepArgs& a, RunWhen when,
                                cudaStream_t st) {
  switch (D) {
    case 1: return launch_dim<1>(density, p, a, when, st);
    case 2: return launch_dim<2>(density, p, a, when, st);
    case 3: return launch_dim<3>(density, p, a, when, st);
    case 4: return launch_dim<4>(density, p, a, when, st);
    case 5: return launch_dim<5>(density, p, a, when, st);
    case 6: return launch_dim<6>(density, p, a, when, st);
    case 7: return launch_dim<7>(density, p, a, when, st);
    case 8: return launch_dim<8>(density, p, a, when, st);
    case 9: return launch_dim<9>(density, p, a, when, st);
    case 10: return launch_dim<10>(density, p, a, when, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace clue_impl
