// sweep_any.cu — local density (core/detail/ClusteringKernels.hpp:29-140) and
// nearest higher (:142-291) off the fast path: any number of dimensions, metric,
// kernel and option, and the choice between the three forms they come in (any_form).
//
// A block of 8 warps takes 32 points of the work order, lane l of every warp
// holding the l-th, and passes over those of one tile together. The tiles of the
// union of their search boxes are walked in the reference's order; the warps take
// 32 of their points each, round by round, and test them against their 32 points.
// For the density every lane leaves its contributions, in order, in shared memory
// and one warp adds them up: a density is a chain of rounded additions in the
// reference's order, but the distances and kernel values are not part of the
// chain. For the nearest higher each warp keeps its best, and the best of the
// warps is the answer: the comparisons are a strict order on (distance, density,
// tag, visiting order).
// With one thread per point over its whole box (sweep_any_thread.cu) an event of
// 32,768 points fills 8 warps on each of the SMs, all
// waiting for their own loads and additions: density and nearest higher took 1.32 +
// 1.42 ms for 32,768 points in 2-D with the periodic metric, 0.17 + 0.14 ms here.
#include <cfloat>
#include <climits>

#include "engine.h"
#include "sweep_device.cuh"

namespace clue_impl {

namespace {

constexpr int kWarps = kThreads / 32;

// Floats per record in shared memory: whole vectors.
template <int D>
constexpr int padded() {
  return D == 1 ? 1 : D == 2 ? 2 : (D + 3) / 4 * 4;
}

// The tiles of the union of the points' search boxes, one per thread at a time,
// and the warps' candidates.
template <int D>
struct Stage {
  int begin[kThreads];    // first sorted position of the tile
  int off[kThreads + 1];  // points of the tiles before it
  int rel[D][kThreads];   // tile coordinates relative to the union box
  __align__(16) float x[kWarps][32][padded<D>()];
  float sig[kWarps][32][D];  // Mahalanobis only
  int scan[kWarps];
};

template <int D>
struct DensityStage : Stage<D> {
  float w[kWarps][32];
  int q[kWarps][32];
  uint8_t count[kWarps][32];
  float add[kWarps][32][32];  // [warp][k][lane]: the lane's k-th contribution of the warp's chunk
};

struct AnyBest {
  float dist, hi;  // no candidate with metric_inner above hi can win
  int q, order;
  uint64_t key;
};

template <int D>
struct NearestStage : Stage<D> {
  uint64_t key[kWarps][32];
  AnyBest best[kWarps][32];
};

// The points of an item, one per lane, alike in every warp, and the passes over
// them. A pass takes the lanes of one tile (`in`), whose boxes are intervals of
// tile coordinates relative to that tile; `lo`/`hi` are the lane's and
// `ulo`/`nu` the union's. In a wrapped dimension the interval runs on past the
// edge, so relative coordinates keep every lane's own visiting order.
template <int D>
struct Item {
  const RunParams& p;
  const SweepArgs& a;
  int s, event;
  EventDesc ev;
  bool active;
  float xi[D], si[D];
  int own[D], lo[D], hi[D];
  bool odd;       // its own tile is not in its box: passes alone
  bool alone;     // this pass is such a lane's
  unsigned todo;
  bool in;
  int ulo[D], nu[D];
  int64_t n_union;
  bool uniform;   // every lane of the pass has the union as its box
  int grid, tile_base;
  int tile[D];    // the pass's tile

  __device__ Item(const RunParams& p, const SweepArgs& a) : p(p), a(a) {}

  __device__ void load(const int32_t* work, int64_t item, float radius) {
    const int lane = threadIdx.x & 31;
    const int64_t w = item * 32 + lane;
    active = w < a.n;
    s = work[active ? w : item * 32];
    event = a.sevt[s];
    ev = a.events[event];
    const GridDesc& g = a.grids[ev.grid];
    load_point<D>(p, a, s, xi, si);
    int inf[D], sup[D];
    search_box<D>(g, p, xi, si, radius, inf, sup);
    odd = false;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      own[d] = get_bin(g, p, xi[d], d);
      // (a box whose ends cross is walked from its lower end as one bin)
      sup[d] = max(sup[d], inf[d]);
      lo[d] = inf[d] - own[d];
      hi[d] = sup[d] - own[d];
      if (p.wrapped[d] && hi[d] >= g.k) {  // the own tile a turn later
        lo[d] -= g.k;
        hi[d] -= g.k;
      }
      odd |= lo[d] > 0 || hi[d] < 0;
    }
    todo = __ballot_sync(kFullMask, active);
  }

  // The next pass's lanes and union. Alike in every warp. (Every shuffle is
  // reached by all lanes.)
  __device__ void next_pass() {
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(todo) - 1;
    const int leader_event = __shfl_sync(kFullMask, event, leader);
    grid = __shfl_sync(kFullMask, ev.grid, leader);
    tile_base = __shfl_sync(kFullMask, ev.tile_base, leader);
    alone = __shfl_sync(kFullMask, (int)odd, leader) != 0;
    in = ((todo >> lane) & 1u) && (alone ? lane == leader : !odd && event == leader_event);
    bool equal = true;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      tile[d] = __shfl_sync(kFullMask, own[d], leader);
      const int l = __shfl_sync(kFullMask, lo[d], leader), h = __shfl_sync(kFullMask, hi[d], leader);
      in &= own[d] == tile[d];
      equal &= lo[d] == l && hi[d] == h;
    }
    const int64_t box = unite();
    // in many dimensions the union of different boxes can hold far more tiles
    // than each: then the lanes with the leader's box only
    const int64_t leader_box = __shfl_sync(kFullMask, box, leader);
    if (n_union > 4 * leader_box + kThreads) {
      in &= equal;
      unite();
    }
    uniform = __all_sync(kFullMask, !in || box == n_union);
    todo &= ~__ballot_sync(kFullMask, in);
  }

  // The union of the boxes of the pass's lanes; returns the tiles of this lane's.
  __device__ int64_t unite() {
    int64_t box = 1;
    n_union = 1;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      ulo[d] = __reduce_min_sync(kFullMask, in ? lo[d] : INT_MAX);
      nu[d] = __reduce_max_sync(kFullMask, in ? hi[d] : INT_MIN) - ulo[d] + 1;
      n_union *= nu[d];
      box *= hi[d] - lo[d] + 1;
    }
    return box;
  }

  // Fills the stage with the union's tiles tb .. tb + 255; returns their points.
  template <typename S>
  __device__ int stage_tiles(S& sh, int64_t tb) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const GridDesc& g = a.grids[grid];
    int m = 0;
    if (tb + tid < n_union) {
      int64_t rem = tb + tid;
      int t = tile_base;
#pragma unroll
      for (int d = D - 1; d >= 0; --d) {
        int r = (int)rem;
        if (d > 0) {
          const int64_t q = n_union < INT_MAX ? (int64_t)((int)rem / nu[d]) : rem / nu[d];
          r = (int)(rem - q * nu[d]);
          rem = q;
        }
        sh.rel[d][tid] = r;
        int b = tile[d] + ulo[d] + r;
        if (p.wrapped[d])
          b = wrap_bin(g, p, b < 0 ? b + 2 * g.k : b, d);
        t += g.stride[d] * b;
      }
      const int begin = a.tile_offset[t];
      m = a.tile_offset[t + 1] - begin;
      sh.begin[tid] = begin;
    }
    int incl = m;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(kFullMask, incl, o);
      if (lane >= o)
        incl += y;
    }
    if (lane == 31)
      sh.scan[warp] = incl;
    __syncthreads();
    int before = 0, total = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      before += w < warp ? sh.scan[w] : 0;
      total += sh.scan[w];
    }
    sh.off[tid] = before + incl - m;
    if (tid == 0)
      sh.off[kThreads] = total;
    __syncthreads();
    return total;
  }

  // The stage's tile that holds stream position pos: the last that starts at or
  // before it (tiles without points share their successor's start).
  template <typename S>
  __device__ static int tile_at(const S& sh, int pos) {
    int k = 0;
#pragma unroll
    for (int o = kThreads / 2; o > 0; o >>= 1)
      k += sh.off[k + o] <= pos ? o : 0;
    return k;
  }

  // The candidates of the warp's chunk that this lane's box holds, from the
  // stage's tile of each lane's candidate (-1: none).
  template <typename S>
  __device__ unsigned accepted(const S& sh, int t_j) const {
    unsigned rest = __ballot_sync(kFullMask, t_j >= 0);
    if (uniform)
      return in ? rest : 0u;
    unsigned acc = 0;
    while (rest) {
      const int t = __shfl_sync(kFullMask, t_j, __ffs(rest) - 1);
      const unsigned run = __ballot_sync(kFullMask, t_j == t);
      bool ok = in;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        const int r = sh.rel[d][t] + ulo[d];
        ok &= lo[d] <= r && r <= hi[d];
      }
      if (ok)
        acc |= run;
      rest &= ~run;
    }
    return acc;
  }
};

// A lane's next candidate, loaded ahead of its use.
template <int D>
struct Candidate {
  int q = -1, t = -1;
  float x[D], sig[D];
};

template <int D, int METRIC, typename S>
__device__ __forceinline__ void fetch(const RunParams& p, const SweepArgs& a, const S& sh, int pos, int total,
                                      Candidate<D>& c) {
  c.q = c.t = -1;
  if (pos < total) {
    c.t = Item<D>::tile_at(sh, pos);
    c.q = sh.begin[c.t] + (pos - sh.off[c.t]);
#pragma unroll
    for (int d = 0; d < D; ++d) {
      c.x[d] = a.sx[d * a.n + c.q];
      if (METRIC == kAnyMetric && p.metric_kind == CLUE_METRIC_MAHALANOBIS)
        c.sig[d] = a.ssig[d * a.n + c.q];
    }
  }
}

template <int D, int METRIC, typename S>
__device__ __forceinline__ void stage_candidate(const RunParams& p, S& sh, int warp, int lane,
                                                const Candidate<D>& c) {
#pragma unroll
  for (int d = 0; d < D; ++d) {
    sh.x[warp][lane][d] = c.x[d];
    if (METRIC == kAnyMetric && p.metric_kind == CLUE_METRIC_MAHALANOBIS)
      sh.sig[warp][lane][d] = c.sig[d];
  }
}

// Distance value of the pair (this lane's point, candidate j of the warp's chunk).
template <int D, int METRIC, typename S>
__device__ __forceinline__ float pair_inner(const RunParams& p, const Item<D>& it, const S& sh, int warp, int j) {
  float xj[padded<D>()], sj[D];
  const float* r = sh.x[warp][j];
  if (padded<D>() == 2) {
    const float2 v = *reinterpret_cast<const float2*>(r);
    xj[0] = v.x, xj[padded<D>() - 1] = v.y;
  } else if (padded<D>() >= 4) {
#pragma unroll
    for (int k = 0; k + 3 < padded<D>(); k += 4) {
      const float4 v = *reinterpret_cast<const float4*>(r + k);
      xj[k] = v.x, xj[k + 1] = v.y, xj[k + 2] = v.z, xj[k + 3] = v.w;
    }
  } else {
    xj[0] = r[0];
  }
  if (METRIC == kAnyMetric)
#pragma unroll
    for (int d = 0; d < D; ++d)
      sj[d] = p.metric_kind == CLUE_METRIC_MAHALANOBIS ? sh.sig[warp][j][d] : 0.0f;
  return inner_distance<D, METRIC>(p, it.xi, xj, it.si, sj);
}

template <int D, int METRIC>
__global__ void __launch_bounds__(kThreads, D <= 4 ? 3 : 2) k_density_any(const RunParams p, const SweepArgs a,
                                                                             const RunWhen when) {
  extern __shared__ __align__(16) unsigned char s_dyn[];
  if (!runs_when(a, when))
    return;
  DensityStage<D>& sh = *reinterpret_cast<DensityStage<D>*>(s_dyn);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t n_items = (a.n + 31) / 32;
  // A candidate out of range adds 0 * k * w: +-0, which leaves a sum as it is,
  // unless k or w is infinite or NaN. Such candidates are evaluated like those in
  // range.
  const float den = __fmul_rn(__fmul_rn(2.0f, p.kernel_p0), p.kernel_p0);
  const bool all_special = !isfinite(p.kernel_p0) || !isfinite(p.kernel_p1) ||
                           (p.kernel_kind == CLUE_KERNEL_GAUSSIAN && !isfinite(den));
  const float thr = metric_has_sqrt(p.metric_kind) ? p.dc2 : p.dc;
  Item<D> it(p, a);
  for (int64_t item = blockIdx.x; item < n_items; item += gridDim.x) {
    it.load(a.work_dens, item, p.dc);
    float rho = 0.0f;
    while (it.todo) {
      it.next_pass();
      for (int64_t tb = 0; tb < it.n_union; tb += kThreads) {
        const int total = it.stage_tiles(sh, tb);
        Candidate<D> next;
        float next_w = 0.0f;
        auto get = [&](int pos) {
          fetch<D, METRIC>(p, a, sh, pos, total, next);
          next_w = next.q >= 0 ? a.sw[next.q] : 0.0f;
        };
        get(threadIdx.x);
        for (int c0 = 0; c0 < total; c0 += kThreads) {
          const int cnt = min(32, total - c0 - warp * 32);
          stage_candidate<D, METRIC>(p, sh, warp, lane, next);
          sh.w[warp][lane] = next_w;
          sh.q[warp][lane] = next.q;
          const unsigned special = __ballot_sync(kFullMask, all_special || !isfinite(next_w));
          const unsigned acc = it.accepted(sh, next.t);
          __syncwarp();
          get(c0 + kThreads + threadIdx.x);
          int k = 0;
          if (__any_sync(kFullMask, acc != 0)) {
            unsigned hit = special;
            if (cnt == 32) {
#pragma unroll 8
              for (int j = 0; j < 32; ++j)
                if (!(pair_inner<D, METRIC>(p, it, sh, warp, j) > thr))
                  hit |= 1u << j;
            } else {
              for (int j = 0; j < cnt; ++j)
                if (!(pair_inner<D, METRIC>(p, it, sh, warp, j) > thr))
                  hit |= 1u << j;
            }
            hit &= acc;
            while (hit) {
              const int j = __ffs(hit) - 1;
              hit &= hit - 1;
              const float dist = metric_finish(p, pair_inner<D, METRIC>(p, it, sh, warp, j));
              const float kv = kernel_value(p, dist, sh.q[warp][j] == it.s);
              // rho_i += static_cast<int>(distance <= density_radius) * k * w_j
              sh.add[warp][k++][lane] = __fmul_rn(__fmul_rn((float)(int)(dist <= p.dc), kv), sh.w[warp][j]);
            }
          }
          sh.count[warp][lane] = (uint8_t)k;
          __syncthreads();
          if (warp == 0) {  // the lanes' sums, in order
            for (int v = 0; v < kWarps; ++v) {
              const int added = sh.count[v][lane];
#pragma unroll 4
              for (int j = 0; j < added; ++j)
                rho = __fadd_rn(rho, sh.add[v][j][lane]);
            }
          }
          __syncthreads();
        }
      }
    }
    if (warp == 0 && it.active) {
      a.srho[it.s] = rho;
      if (a.out_rho)
        a.out_rho[a.perm[it.s]] = rho;
    }
  }
}

template <int D, int METRIC>
__global__ void __launch_bounds__(kThreads, D <= 4 ? 3 : 2) k_nearest_higher_any(const RunParams p, const SweepArgs a,
                                                                                    const RunWhen when) {
  extern __shared__ __align__(16) unsigned char s_dyn[];
  if (!runs_when(a, when))
    return;
  NearestStage<D>& sh = *reinterpret_cast<NearestStage<D>*>(s_dyn);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t n_items = (a.n + 31) / 32;
  const bool root = metric_has_sqrt(p.metric_kind);
  Item<D> it(p, a);
  for (int64_t item = blockIdx.x; item < n_items; item += gridDim.x) {
    it.load(a.work_nh, item, p.dm);
    const int s = it.s, gi = a.perm[s];
    const float rho_i = a.srho[s];
    const float unc = p.has_unc ? a.sunc[s] : 1.0f;
    const float min_density = __fmul_rn(p.rhoc, unc);
    const bool seedlike = rho_i >= min_density;
    // ClusteringKernels.hpp:168; as a bound on metric_inner
    const float eff = seedlike ? p.seed_dc : p.dm;
    const float eff_inner = root ? (seedlike ? p.seed2 : p.dm2) : eff;
    // ClusteringKernels.hpp:180-182 as one order on (density, tag): see rho_key;
    // equal densities count only above zero, else the tag part is saturated
    const bool nan_i = rho_i != rho_i;
    const uint32_t tag_i = p.has_tags ? a.stag[s] : (uint32_t)gi;
    const uint64_t key_i = ((uint64_t)(nan_i ? 0xffffffffu : rho_key(rho_i)) << 32) |
                           ((nan_i || !(rho_i > 0.0f)) ? 0xffffffffu : tag_i);
    // no candidate at FLT_MAX or beyond is taken (the reference starts from there)
    AnyBest best{FLT_MAX, INFINITY, -1, 0, ~0ull};
    auto consider = [&](float inner, uint64_t key, int q, int order) {
      const float dist = metric_finish(p, inner);
      // ClusteringKernels.hpp:195-202
      if (dist <= eff &&
          ((dist < best.dist) ||
           ((dist == best.dist) && ((key > best.key) || (key == best.key && order < best.order))))) {
        // a larger root needs a square larger by 2^-23 relative; tiny squares stay open
        best = AnyBest{dist, !root ? inner : inner >= 0x1p-100f ? __fmul_rn(inner, 1.00000095367431640625f) : INFINITY,
                       q, order, key};
      }
    };
    while (it.todo) {
      it.next_pass();
      int order0 = 0;  // points of the earlier tiles
      for (int64_t tb = 0; tb < it.n_union; tb += kThreads) {
        const int total = it.stage_tiles(sh, tb);
        Candidate<D> next;
        uint64_t next_key = 0;
        auto get = [&](int pos) {
          fetch<D, METRIC>(p, a, sh, pos, total, next);
          if (next.q >= 0)
            next_key = ((uint64_t)rho_key(a.srho[next.q]) << 32) |
                       (p.has_tags ? a.stag[next.q] : (uint32_t)a.perm[next.q]);
        };
        get(threadIdx.x);
        for (int c0 = 0; c0 < total; c0 += kThreads) {
          const int cnt = min(32, total - c0 - warp * 32);
          const int t_j = next.t, q_j = next.q;
          stage_candidate<D, METRIC>(p, sh, warp, lane, next);
          sh.key[warp][lane] = next_key;
          const unsigned acc = it.accepted(sh, t_j);
          __syncwarp();
          get(c0 + kThreads + threadIdx.x);
          const float most = fminf(eff_inner, best.hi);
          unsigned hit = 0;
          if (__any_sync(kFullMask, acc != 0)) {
#pragma unroll 4
            for (int j = 0; j < cnt; ++j)
              if (sh.key[warp][j] > key_i && pair_inner<D, METRIC>(p, it, sh, warp, j) <= most)
                hit |= 1u << j;
          }
          hit &= acc;
          while (__any_sync(kFullMask, hit != 0)) {
            const int j = hit ? __ffs(hit) - 1 : 0;
            const int q = __shfl_sync(kFullMask, q_j, j);
            if (hit)
              consider(pair_inner<D, METRIC>(p, it, sh, warp, j), sh.key[warp][j], q,
                       order0 + c0 + warp * 32 + j);
            hit &= hit - 1;
          }
          __syncwarp();
        }
        order0 += total;
        __syncthreads();  // the stage is rewritten
      }
    }
    // the best of the warps
    sh.best[warp][lane] = best;
    __syncthreads();
    if (warp == 0 && it.active) {
      for (int v = 1; v < kWarps; ++v) {
        const AnyBest b = sh.best[v][lane];
        if (b.q >= 0 &&
            ((b.dist < best.dist) ||
             ((b.dist == best.dist) && ((b.key > best.key) || (b.key == best.key && b.order < best.order)))))
          best = b;
      }
      const int nh = best.q >= 0 ? a.perm[best.q] : -1;
      a.out_nh[gi] = nh;
      a.parent[s] = best.q >= 0 ? best.q : s;
      // KernelFindClusters, ClusteringKernels.hpp:301-313
      const int seed = (nh == -1) && seedlike;
      a.seed_flag[gi] = seed;
      if (a.out_seed)
        a.out_seed[gi] = seed;
    }
    __syncthreads();  // sh.best is rewritten
  }
}

template <int D, int METRIC>
cudaError_t launch_any(bool density, const RunParams& p, const SweepArgs& a, RunWhen when, cudaStream_t st) {
  const int64_t items = (a.n + 31) / 32;
  const int blocks = (int)std::min<int64_t>(items, (int64_t)sm_count() * 64);
  // up to 70 KB: above the default 48 KB they need the opt-in, a function
  // attribute (not stream work: it may come during a capture)
  if (density) {
    constexpr int smem = (int)sizeof(DensityStage<D>);
    const cudaError_t e = cudaFuncSetAttribute(k_density_any<D, METRIC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess)
      return e;
    k_density_any<D, METRIC><<<blocks, kThreads, smem, st>>>(p, a, when);
  } else {
    constexpr int smem = (int)sizeof(NearestStage<D>);
    const cudaError_t e =
        cudaFuncSetAttribute(k_nearest_higher_any<D, METRIC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess)
      return e;
    k_nearest_higher_any<D, METRIC><<<blocks, kThreads, smem, st>>>(p, a, when);
  }
  count_launches(1);
  return cudaGetLastError();
}

template <int D>
cudaError_t launch_dim(bool density, const RunParams& p, const SweepArgs& a, RunWhen when, cudaStream_t st) {
  switch (p.metric_kind) {
    case CLUE_METRIC_EUCLIDEAN: return launch_any<D, CLUE_METRIC_EUCLIDEAN>(density, p, a, when, st);
    case CLUE_METRIC_PERIODIC_EUCLIDEAN: return launch_any<D, CLUE_METRIC_PERIODIC_EUCLIDEAN>(density, p, a, when, st);
    default: return launch_any<D, kAnyMetric>(density, p, a, when, st);
  }
}

cudaError_t launch_sweep_block(bool density, int D, const RunParams& p, const SweepArgs& a, RunWhen when,
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

cudaError_t launch_forms(bool density, int D, const RunParams& p, const SweepArgs& a, cudaStream_t st) {
  const AnyForm f = any_form(D, a);
  cudaError_t e = cudaSuccess;
  if (f.point)
    e = launch_sweep_point(density, D, p, a, st);
  if (e == cudaSuccess && f.block)
    e = launch_sweep_block(density, D, p, a, f.block, st);
  if (e == cudaSuccess && f.thread)
    e = launch_sweep_thread(density, D, p, a, f.thread, st);
  return e;
}

}  // namespace

// The form of a run's sweeps. A thread per point takes as long as its longest chain of
// candidates, about 0.35 us each, until the points fill the GPU; the other forms take
// a time that grows with the number of points (a block of 32 points of one tile about
// 0.75 ns a point and more where a tile holds fewer) and little with the candidates.
// Few candidates: events of few points. Density + nearest higher, us, thread / warp
// per point, 16,384 points in events of 16: 22 / 40, 32: 33 / 38, 64: 49 / 42, 256:
// 174 / 54; thread / block, 32,768 points in events of 64: 49 / 66, 128: 84 / 67;
// 65,536 in events of 128: 90 / 104, 256: 186 / 141; 131,072 in events of 256: 217 / 250.
// Tiles of few points: one grid for a batch, 65,536 points in 32 events of 2,048 (4
// points a tile) 184 / 592, in 4-D 274 / 606; per event, 65,536 in 4-D events of 256 (16
// points a tile) 172 / 317, of 512 (32) 289 / 300.
// But one event of sparse tiles in many dimensions has many candidates (a call, thread /
// block): 16,385 points in 6-D (22 a tile) 425 / 258 and 1,415 / 654, 65,536 in 7-D (30)
// 778 / 717 and 4,096 / 3,287, in 8-D (10) 675 / 848 (24 a tile asked for, 65,536 in 2-D 466 /
// 534, 3-D 471 / 633, 4-D 642 / 791); above that many points the threads fill the GPU:
// 110,000 in 6-D (27 a tile) 1,718 / 2,074, 131,072 in 6-D (32) 972 / 1,120 and 2,934 / 4,237,
// but 90,000 in 6-D (123) 4,846 / 2,656.
// Beyond 65,536 points it depends on the points. Even ones (no tile of more than 256
// points) in one event, dc of 0.05 and 0.3 tiles, a call, thread / block: 70,000 in 1-D 326 /
// 253 and 336 / 299, in 3-D 646 / 445 and 714 / 722, in 5-D 1,043 / 677 and 2,475 / 1,671;
// 100,000 in 1-D 340 / 283 and 349 / 344, in 3-D 696 / 574 and 795 / 953, in 4-D 985 / 618
// and 1,504 / 1,316; 131,072 in 3-D 696 / 675 and 875 / 1,191, in 4-D 1,329 / 828 and 2,122 /
// 1,916, in 7-D 1,750 / 1,889 and 10,164 / 9,271; 200,000 in 5-D 1,500 / 1,579 and 4,173 /
// 4,538. Clustered ones of 131,072 in 4-D 3,546 / 1,153, 262,144 in 1-D 1,852 / 1,612;
// 1,048,576 in 2-D 8,149 / 6,860, in 3-D 8,784 / 7,120, but in 1-D 4,717 / 6,147. So both
// kernels are launched there, and in smaller runs of sparse tiles, and one of them returns
// at once (about 4 us).
AnyForm any_form(int D, const SweepArgs& a) {
  constexpr int64_t kPointWarps = 1 << 14, kBlocks = 1 << 16;
  const bool one = a.n_events <= 1;
  const int64_t even_blocks = !one ? kBlocks : D <= 3 ? 5 << 14 : 1 << 17;
  const int64_t most_blocks = D == 1 ? 1 << 18 : 1 << 20;
  AnyForm f;
  const int64_t event = std::min<int64_t>(a.n / std::max(1, a.n_events), 512);  // points, at most 512
  const int tile = a.n > kBlocks ? 48 : one && D >= 6 ? 16 : 32;  // points
  const bool few = a.n > 256 * event, sparse = a.n < tile * a.n_tiles;
  if (a.n <= kPointWarps) {
    (few ? f.thread : f.point) = kAlways;
    return f;
  }
  f.work_order = true;
  if (a.n <= even_blocks && !few && !sparse) {
    f.block = kAlways;
  } else if (a.n <= most_blocks && a.max_event_points > kLargeTilePoints) {
    f.block = kLargeTiles;
    f.thread = kNoLargeTiles;
  } else {  // (no tile can hold more than 256 points, or the points fill the GPU)
    f.thread = kAlways;
  }
  return f;
}

cudaError_t launch_density_any(int D, const RunParams& p, const SweepArgs& a, cudaStream_t st) {
  return launch_forms(true, D, p, a, st);
}

cudaError_t launch_nearest_higher_any(int D, const RunParams& p, const SweepArgs& a, cudaStream_t st) {
  return launch_forms(false, D, p, a, st);
}

}  // namespace clue_impl
