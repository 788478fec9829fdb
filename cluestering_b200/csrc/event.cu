// event.cu — single events of at most kEventPoints points: everything before
// the sweeps in one launch (k_event_front) and everything after them in another
// (k_event_finish), each by one thread-block cluster whose blocks exchange
// their partial results through distributed shared memory.
//
// The general pipeline takes 11 launches before the sweeps and 4 after them,
// most of them one or two blocks on an event this small, each a few
// microseconds of launch and memory latency; its stable binning runs one warp
// per 1,024 points and its label kernel one block per event. Measured on B200
// (16,384-point 2-D event, sums of kernel times): 153 us before the sweeps and
// 45 us after them there, 14 us and 16 us here.
#include <atomic>
#include <cfloat>
#include <type_traits>

#include <cooperative_groups.h>

#include "engine.h"
#include "sweep.cuh"

namespace clue_impl {

namespace {

namespace cg = cooperative_groups;

constexpr unsigned kFull = 0xffffffffu;
constexpr int kBlock = 1024;
constexpr int kWarps = kBlock / 32;
constexpr int kMaxCluster = 16;  // above 8 the kernels need the opt-in (event_path)
// Rounds of 32 points per warp at the largest event and cluster.
constexpr int kRounds = kEventPoints / (kMaxCluster * kBlock);

struct FrontArgs {
  const float* x[kMaxDim];
  const float* sig[kMaxDim];
  const float* weight;
  const float* unc;
  const uint32_t* tags;
  GridDesc grid;  // shape only; the extents come from the points
  EventDesc ev;
  GridDesc* grids;
  EventDesc* events;
  int32_t* point_event;
  int32_t* tile_offset;
  int32_t* perm;
  int32_t* sevt;
  float* sx;
  float* sw;
  float* ssig;
  float* sunc;
  uint32_t* stag;
  float4* rec;  // density records of the fast sweeps, or null
  int32_t* event_exact;  // or null
  int32_t* counters;
  int32_t* large_count;  // tiles of more than kLargeTilePoints points (any_form), or null
};

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Exclusive prefix of v over the block's threads; *total = the block's sum.
__device__ __forceinline__ int block_exclusive(int v, int* s_warp, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(kFull, incl, o);
    if (lane >= o)
      incl += y;
  }
  if (lane == 31)
    s_warp[warp] = incl;
  __syncthreads();
  const int w = s_warp[lane];  // one entry per warp: 32 of them
  int wi = w;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(kFull, wi, o);
    if (lane >= o)
      wi += y;
  }
  *total = __shfl_sync(kFull, wi, 31);
  const int before = __shfl_sync(kFull, wi - w, warp);
  __syncthreads();  // s_warp may be reused
  return before + incl - v;
}

// A stable counting sort of up to C * kBlock * kRounds keys by the blocks of a
// cluster. Every warp owns a run of consecutive elements. It counts them per key
// in its own column of shared counters; the columns become prefixes over the
// block's warps and, through the blocks' totals, over the cluster; then the warp
// places its elements in order. Equal keys therefore stay in index order.
struct ClusterSort {
  int* tot;       // elements of each key in this block (read by the others)
  int* base;      // first position of this block's elements of a key
  uint16_t* all;  // [kWarps][Kp]: counts, then prefixes over the warps
  uint16_t* col;  // this warp's column
  int Kp;

  __device__ ClusterSort(unsigned char* smem, int keys) {
    Kp = (keys + 1) & ~1;
    tot = reinterpret_cast<int*>(smem);
    base = tot + Kp;
    all = reinterpret_cast<uint16_t*>(base + Kp);
    col = all + (threadIdx.x >> 5) * Kp;
  }
  static size_t bytes(int keys) {
    return (size_t)((keys + 1) & ~1) * (2 * sizeof(int) + kWarps * sizeof(uint16_t));
  }
  // Clears the counters (a block barrier must follow).
  __device__ void clear() {
    for (int k = threadIdx.x; k < kWarps * Kp / 2; k += kBlock)
      reinterpret_cast<uint32_t*>(all)[k] = 0;
  }
  // Counts the warp's next 32 elements (key < 0: none on this lane).
  __device__ void count(int key) {
    const unsigned mask = __match_any_sync(kFull, key);
    if (key >= 0 && (int)(threadIdx.x & 31) == __ffs(mask) - 1)
      col[key] += (uint16_t)__popc(mask);
    __syncwarp();  // the next round's leaders read these counters
  }
  // Prefixes over the block's warps and the block's totals (barriers before and
  // after, the latter a cluster barrier).
  __device__ void block_prefix(int keys) {
    for (int k = threadIdx.x; k < keys; k += kBlock) {
      int run = 0;
#pragma unroll 8
      for (int w = 0; w < kWarps; ++w) {
        const int v = all[w * Kp + k];
        all[w * Kp + k] = (uint16_t)run;
        run += v;
      }
      tot[k] = run;
    }
  }
  // Bases of this block's elements, from the totals of every block, and the
  // first position of every key, which block 0 hands to emit(key, first, elements).
  // Returns the number of elements. The others' shared memory has been read
  // when it returns.
  template <typename Emit>
  __device__ int bases(cg::cluster_group& cluster, int keys, int* s_warp, Emit&& emit) {
    const int C = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int per = (keys + kBlock - 1) / kBlock;  // consecutive keys per thread
    const int k0 = min(keys, (int)threadIdx.x * per), k1 = min(keys, k0 + per);
    int counts[kKeysPerThread];
    int mine = 0;
#pragma unroll
    for (int j = 0; j < kKeysPerThread; ++j) {
      counts[j] = 0;
      if (k0 + j < k1) {
        int before = 0;
#pragma unroll 4
        for (int q = 0; q < C; ++q) {
          const int v = cluster.map_shared_rank(tot, q)[k0 + j];
          counts[j] += v;
          before += q < rank ? v : 0;
        }
        base[k0 + j] = mine + before;
        mine += counts[j];
      }
    }
    int total;
    int first = block_exclusive(mine, s_warp, &total);
    const int block_first = first;
#pragma unroll
    for (int j = 0; j < kKeysPerThread; ++j)
      if (k0 + j < k1) {
        base[k0 + j] += block_first;
        if (rank == 0)
          emit(k0 + j, first, counts[j]);
        first += counts[j];
      }
    return total;
  }
  // Position of this lane's element of the warp's next 32, in the order of count().
  __device__ int place(int key) {
    const unsigned mask = __match_any_sync(kFull, key);
    const int leader = __ffs(mask) - 1;
    int at = 0;
    if (key >= 0 && (int)(threadIdx.x & 31) == leader) {
      at = col[key];
      col[key] = (uint16_t)(at + __popc(mask));
    }
    at = __shfl_sync(kFull, at, leader);
    __syncwarp();
    return key < 0 ? -1 : base[key] + at + __popc(mask & lanemask_lt());
  }
  static constexpr int kKeysPerThread = (kEventTiles + kBlock - 1) / kBlock;
};

// Extents, tile binning and the tile-contiguous copy of one event: its points
// sorted by tile with ClusterSort, so every tile lists them in ascending index
// (AssociationMap.hpp:63-81). Bound by latency: one round of global loads (in
// 2-D and 3-D every coordinate stays in registers, all rounds loaded at once),
// three cluster barriers and the scattered stores.
// DD: 2 or 3 dimensions, or 0 for any number.
template <int DD>
__global__ void __launch_bounds__(kBlock, 1) k_event_front(const RunParams p, const FrontArgs a) {
  extern __shared__ __align__(16) unsigned char s_dyn[];
  __shared__ GridDesc sg;
  __shared__ float s_red[2 * kMaxDim][kWarps];
  __shared__ float s_ext[2 * kMaxDim];  // this block's extremes (read by the others)
  __shared__ int s_sum[4];              // this block's exact-sum bounds (idem)
  __shared__ int s_warp[kWarps];
  cg::cluster_group cluster = cg::this_cluster();
  const int C = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int D = DD ? DD : p.D;
  const int n = a.ev.n, T = a.grid.T;
  ClusterSort sort(s_dyn, T);
  // the warp's run of points: a multiple of 32 of them
  const int per_warp = ((n + C * kWarps - 1) / (C * kWarps) + 31) & ~31;
  const int begin = min(n, (rank * kWarps + warp) * per_warp), end = min(n, begin + per_warp);

  if (threadIdx.x < 4)
    s_sum[threadIdx.x] = threadIdx.x == 0 ? INT_MAX : 0;
  if (threadIdx.x == 0)
    sg = a.grid;
  if (a.large_count && rank == 0 && threadIdx.x == 0)
    *a.large_count = 0;
  float x[kRounds][DD ? DD : 1], w[kRounds];
#pragma unroll
  for (int k = 0; k < kRounds; ++k) {
    const int i = begin + k * 32 + lane;
#pragma unroll
    for (int d = 0; d < DD; ++d)
      x[k][d] = i < end ? a.x[d][i] : 0.0f;
    w[k] = i < end ? a.weight[i] : 0.0f;
  }
  sort.clear();

  // ---- extents (ComputeTiles.hpp:16-62) ----
#pragma unroll
  for (int d = 0; d < (DD ? DD : kMaxDim); ++d) {
    if (d >= D)
      break;
    float mn = FLT_MAX, mx = -FLT_MAX;
#pragma unroll
    for (int k = 0; k < kRounds; ++k) {
      const int i = begin + k * 32 + lane;
      if (i < end) {
        const float v = DD ? x[k][DD ? d : 0] : a.x[d][i];
        if (v == v) {  // NaN never becomes an extreme
          mn = fminf(mn, v);
          mx = fmaxf(mx, v);
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      mn = fminf(mn, __shfl_xor_sync(kFull, mn, o));
      mx = fmaxf(mx, __shfl_xor_sync(kFull, mx, o));
    }
    if (lane == 0) {
      s_red[2 * d][warp] = mn;
      s_red[2 * d + 1][warp] = mx;
    }
  }
  __syncthreads();
  if (warp < D) {
    float mn = s_red[2 * warp][lane], mx = s_red[2 * warp + 1][lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      mn = fminf(mn, __shfl_xor_sync(kFull, mn, o));
      mx = fmaxf(mx, __shfl_xor_sync(kFull, mx, o));
    }
    if (lane == 0) {
      s_ext[2 * warp] = mn;
      s_ext[2 * warp + 1] = mx;
    }
  }
  cluster.sync();
  if (warp < D) {  // lane q: the extremes of block q
    float mn = FLT_MAX, mx = -FLT_MAX;
    if (lane < C) {
      const float* e = cluster.map_shared_rank(s_ext, lane);
      mn = e[2 * warp];
      mx = e[2 * warp + 1];
    }
#pragma unroll
    for (int o = kMaxCluster / 2; o > 0; o >>= 1) {
      mn = fminf(mn, __shfl_xor_sync(kFull, mn, o));
      mx = fmaxf(mx, __shfl_xor_sync(kFull, mx, o));
    }
    if (lane == 0) {
      sg.minv[warp] = mn;
      sg.maxv[warp] = mx;
      sg.tile[warp] = __fdiv_rn(__fsub_rn(mx, mn), (float)sg.k);
    }
  }
  __syncthreads();
  if (rank == 0 && threadIdx.x == 0) {
    a.grids[0] = sg;
    a.events[0] = a.ev;
  }

  // ---- tile of every point ----
  const bool bounds = a.event_exact && p.kernel_kind == CLUE_KERNEL_FLAT;  // uniform
  int lsb = INT_MAX, bad = 0;
  uint32_t vb = 0, wb = 0;
  int tile[kRounds];
#pragma unroll
  for (int k = 0; k < kRounds; ++k) {
    const int i = begin + k * 32 + lane;
    tile[k] = -1;
    if (i < end) {
      int t = 0;
#pragma unroll
      for (int d = 0; d < (DD ? DD : kMaxDim); ++d)
        if (d < D)
          t += sg.stride[d] * get_bin(sg, p, DD ? x[k][DD ? d : 0] : a.x[d][i], d);
      tile[k] = t;
      if (bounds) {
        const float v = __fmul_rn(p.kernel_p0, w[k]);  // a neighbour's fl(flat * w_j)
        const int bd = !(w[k] >= 0.0f) || signbit(w[k]) || isinf(w[k]) || isinf(v);
        bad |= bd;
        if (!bd) {
          if (v > 0.0f)
            lsb = min(lsb, lsb_exponent(v));
          if (w[k] > 0.0f)
            lsb = min(lsb, lsb_exponent(w[k]));
          vb = max(vb, __float_as_uint(v));
          wb = max(wb, __float_as_uint(w[k]));
        }
      }
    }
    if (begin + k * 32 < end)  // warp-uniform
      sort.count(tile[k]);
  }
  if (bounds) {
    lsb = __reduce_min_sync(kFull, lsb);
    vb = __reduce_max_sync(kFull, vb);
    wb = __reduce_max_sync(kFull, wb);
    bad = __any_sync(kFull, bad);
    if (lane == 0) {
      atomicMin(&s_sum[0], lsb);
      atomicMax(reinterpret_cast<unsigned*>(&s_sum[1]), vb);
      atomicMax(reinterpret_cast<unsigned*>(&s_sum[2]), wb);
      atomicOr(&s_sum[3], bad);
    }
  }
  __syncthreads();
  sort.block_prefix(T);
  cluster.sync();

  // ---- tile offsets, and where this block's points of each tile start ----
  if (rank == 0 && threadIdx.x == kBlock - 1) {
    if (a.event_exact) {
      int4 st = make_int4(INT_MAX, 0, 0, 0);
      for (int q = 0; q < C; ++q) {
        const int* b = cluster.map_shared_rank(s_sum, q);
        st.x = min(st.x, b[0]);
        st.y = max(st.y, b[1]);  // non-negative floats: their bits order like ints
        st.z = max(st.z, b[2]);
        st.w |= b[3];
      }
      reinterpret_cast<int4*>(a.event_exact)[0] = st;
    }
    a.counters[4] = a.counters[5] = 0;   // the sweeps' work queues
    a.counters[9] = a.counters[10] = 0;  // SweepArgs::load
  }
  sort.bases(cluster, T, s_warp, [&](int t, int first, int count) {
    a.tile_offset[t] = first;
    if (a.large_count && count > kLargeTilePoints)
      atomicAdd(a.large_count, 1);
  });
  // the others' shared memory has been read: after the matching wait at the
  // end every block may exit
  __syncwarp();
  cluster.barrier_arrive();
  __syncthreads();
  if (rank == 0 && threadIdx.x == 0)
    a.tile_offset[T] = n;

  // ---- placement and the tile-contiguous copy ----
#pragma unroll
  for (int k = 0; k < kRounds; ++k) {
    if (begin + k * 32 >= end)
      continue;  // warp-uniform
    const int i = begin + k * 32 + lane;
    const int64_t s = sort.place(tile[k]);
    if (s < 0)
      continue;
    a.sevt[i] = 0;
    a.point_event[i] = 0;
    // The stores are scattered, and 16 SMs make them all: as few as possible. The
    // event of every position is the same, and where the sweeps read records
    // nothing reads the coordinate planes.
    a.perm[s] = i;
    a.sw[s] = w[k];
    if (!(DD && a.rec)) {
#pragma unroll
      for (int d = 0; d < (DD ? DD : kMaxDim); ++d)
        if (d < D)
          a.sx[(int64_t)d * n + s] = DD ? x[k][DD ? d : 0] : a.x[d][i];
    } else {  // {x, y, v, w} or {x, y, z, v}, as k_gather writes them
      const float v = p.kernel_kind == CLUE_KERNEL_FLAT ? __fmul_rn(p.kernel_p0, w[k]) : w[k];
      a.rec[s] = DD == 2 ? make_float4(x[k][0], x[k][DD ? 1 : 0], v, w[k])
                         : make_float4(x[k][0], x[k][DD ? 1 : 0], x[k][DD == 3 ? 2 : 0], v);
    }
    if (p.has_sigma)
      for (int d = 0; d < D; ++d)
        a.ssig[(int64_t)d * n + s] = ((p.has_sigma >> d) & 1) ? a.sig[d][i] : 0.0f;
    if (a.unc)
      a.sunc[s] = a.unc[i];
    if (a.tags)
      a.stag[s] = a.tags[i];
  }
  __syncwarp();
  cluster.barrier_wait();
}

// Cluster -> points map (utils/detail/get_clusters.hpp:24-49): a stable counting
// sort of the points by label. Outliers (-1) are left out, and so is any label that is
// not below n_clusters: the labels are the caller's memory, which may have been written
// since the run, and here they index shared memory. One launch for the nine
// of the general form (histogram, scan, scatter and the ordering of each
// cluster's ids): 45 -> 7 us for 32,768 points in 40 clusters.
__global__ void __launch_bounds__(kBlock, 1) k_event_map(int n, const int32_t* labels, int n_clusters,
                                                         int32_t* offsets, int32_t* points) {
  extern __shared__ __align__(16) unsigned char s_dyn[];
  __shared__ int s_warp[kWarps];
  cg::cluster_group cluster = cg::this_cluster();
  const int C = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  ClusterSort sort(s_dyn, n_clusters);
  const int per_warp = ((n + C * kWarps - 1) / (C * kWarps) + 31) & ~31;
  const int begin = min(n, (rank * kWarps + warp) * per_warp), end = min(n, begin + per_warp);
  int label[kRounds];
#pragma unroll
  for (int k = 0; k < kRounds; ++k) {
    const int i = begin + k * 32 + lane;
    const int l = i < end ? labels[i] : -1;
    label[k] = (unsigned)l < (unsigned)n_clusters ? l : -1;
  }
  sort.clear();
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kRounds; ++k)
    if (begin + k * 32 < end)  // warp-uniform
      sort.count(label[k]);
  __syncthreads();
  sort.block_prefix(n_clusters);
  cluster.sync();
  const int total = sort.bases(cluster, n_clusters, s_warp, [&](int c, int first, int) { offsets[c] = first; });
  __syncwarp();
  cluster.barrier_arrive();
  __syncthreads();
  if (rank == 0 && threadIdx.x == 0)
    offsets[n_clusters] = total;
#pragma unroll
  for (int k = 0; k < kRounds; ++k)
    if (begin + k * 32 < end) {
      const int s = sort.place(label[k]);
      if (s >= 0)
        points[s] = begin + k * 32 + lane;
    }
  __syncwarp();
  cluster.barrier_wait();
}

// Cluster ids of one event: the seeds ranked in index order (a scan over the
// cluster's blocks), then the root of every point's follower chain. Each block
// copies the event's whole follower tree into its shared memory as 16-bit
// positions (up to 128 KB) and its threads walk their own points' chains there;
// no step leaves the SM. The same outputs as k_scan over the seed flags and
// k_labels.
__global__ void __launch_bounds__(kBlock, 1)
    k_event_finish(int n, const int32_t* parent, const int32_t* perm, const int32_t* seed_flag,
                   int32_t* seed_rank, int32_t* cluster_index, int32_t* seeds, int32_t* seed_event,
                   int32_t* n_seeds, uint32_t* status, int32_t* host_n_seeds, uint32_t* host_status) {
  extern __shared__ __align__(16) uint16_t up[];
  __shared__ int s_warp[kWarps];
  __shared__ int s_total;  // this block's seeds (read by the others)
  cg::cluster_group cluster = cg::this_cluster();
  const int C = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  // the thread's run of consecutive points, and its positions in the layout
  const int per = (n + C * kBlock - 1) / (C * kBlock);
  const int b = min(n, (rank * kBlock + (int)threadIdx.x) * per), e = min(n, b + per);
  int flags = 0;
#pragma unroll
  for (int k = 0; k < kRounds; ++k)
    if (b + k < e)
      flags |= (seed_flag[b + k] ? 1 : 0) << k;
  int root[kRounds], gi[kRounds];
#pragma unroll
  for (int k = 0; k < kRounds; ++k) {
    const int s = (k * C + rank) * kBlock + threadIdx.x;
    root[k] = s < n ? s : -1;
    gi[k] = s < n ? perm[s] : 0;
  }
  bool outside = false;
#pragma unroll 8
  for (int s = threadIdx.x; s < n; s += kBlock) {
    const unsigned q = (unsigned)parent[s];
    up[s] = (uint16_t)(q < (unsigned)n ? q : (unsigned)s);
    outside |= q >= (unsigned)n;
  }
  if (outside)  // a chain leaving its event: never
    atomicOr(status, kStatusLabelRange);
  int total;
  int at = block_exclusive(__popc(flags), s_warp, &total);
  if (threadIdx.x == 0)
    s_total = total;
  cluster.sync();
  int all = 0;
  for (int q = 0; q < C; ++q) {
    const int v = *cluster.map_shared_rank(&s_total, q);
    at += q < rank ? v : 0;
    all += v;
  }
#pragma unroll
  for (int k = 0; k < kRounds; ++k)
    if (b + k < e) {
      seed_rank[b + k] = at;
      if ((flags >> k) & 1) {
        seeds[at] = b + k;
        seed_event[at] = 0;
        ++at;
      }
    }
  // All of the thread's chains at once, so that their steps overlap, each step
  // leaving its point on its grandparent: every write stores an ancestor, so
  // the threads' walks shorten each other's. Where some chain is still longer
  // after kWalk steps, a round over the whole tree at least halves every path.
  constexpr int kWalk = 32;
  for (int round = 0;; ++round) {
    bool moved = true;
    for (int step = 0; step < kWalk && moved; ++step) {
      moved = false;
#pragma unroll
      for (int k = 0; k < kRounds; ++k)
        if (root[k] >= 0) {
          const int q = up[root[k]];
          const int qq = up[q];
          if (qq != q)
            up[root[k]] = (uint16_t)qq;
          moved |= qq != root[k];
          root[k] = qq;
        }
    }
    if (!__syncthreads_or(moved))
      break;
    if (round > 16) {  // a cycle: never (16 rounds shorten 65,536 steps to one)
      atomicOr(status, kStatusLabelTimeout);
      break;
    }
#pragma unroll 8
    for (int s = threadIdx.x; s < n; s += kBlock)
      up[s] = up[up[s]];
    __syncthreads();
  }
  // every seed rank is written before any block reads one (and the totals have
  // been read)
  cluster.sync();
  int gr[kRounds], flag[kRounds];
#pragma unroll
  for (int k = 0; k < kRounds; ++k)
    gr[k] = root[k] >= 0 ? perm[root[k]] : -1;
#pragma unroll
  for (int k = 0; k < kRounds; ++k)
    flag[k] = gr[k] >= 0 ? seed_flag[gr[k]] : 0;
#pragma unroll
  for (int k = 0; k < kRounds; ++k)
    if (gr[k] >= 0)
      cluster_index[gi[k]] = flag[k] ? __ldcg(&seed_rank[gr[k]]) : -1;
  if (host_n_seeds)  // the status word is read after every block's last write to it
    cluster.sync();
  if (rank == 0 && threadIdx.x == 0) {
    *n_seeds = all;
    if (host_n_seeds) {  // pinned host memory: read by the host once the run has finished
      *host_n_seeds = all;
      *host_status = atomicOr(status, 0u);
    }
  }
}

// Blocks of the cluster: a point per thread as far as the largest cluster goes,
// so that small events pay for small barriers only and larger ones use more SMs.
int cluster_blocks(int64_t n) {
  int C = 1;
  while (C < kMaxCluster && (int64_t)C * kBlock < n)
    C *= 2;
  return C;
}

size_t finish_smem(int64_t n) { return ((size_t)n * sizeof(uint16_t) + 15) & ~(size_t)15; }

const cudaLaunchConfig_t* cluster_config(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr, int C, size_t smem,
                                         cudaStream_t st) {
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = C;
  attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
  cfg->gridDim = dim3(C);
  cfg->blockDim = dim3(kBlock);
  cfg->dynamicSmemBytes = smem;
  cfg->stream = st;
  cfg->attrs = attr;
  cfg->numAttrs = 1;
  return cfg;
}

template <typename... Args>
cudaError_t launch_cluster(void (*kernel)(Args...), int C, size_t smem, cudaStream_t st,
                           std::common_type_t<Args>... args) {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr{};
  count_launches(1);
  return cudaLaunchKernelEx(cluster_config(&cfg, &attr, C, smem, st), kernel, args...);
}

}  // namespace

// Grants the kernels their shared memory (above the default 48 KB) and cluster
// size (above 8) on the current device, once per device; false where it
// refuses either.
static bool clusters_ready() {
  constexpr int kDevices = 64;
  static std::atomic<int> granted[kDevices];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices)
    return false;
  int state = granted[dev].load(std::memory_order_relaxed);
  if (state == 0) {
    const auto grant = [](auto kernel, size_t smem) {
      cudaLaunchConfig_t cfg{};
      cudaLaunchAttribute attr{};
      int clusters = 0;
      return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess &&
             cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
             cudaOccupancyMaxActiveClusters(&clusters, kernel, cluster_config(&cfg, &attr, kMaxCluster, smem, 0)) ==
                 cudaSuccess &&
             clusters >= 1;
    };
    const size_t sort = ClusterSort::bytes(kEventTiles);
    const bool ok = grant(k_event_front<0>, sort) && grant(k_event_front<2>, sort) && grant(k_event_front<3>, sort) &&
                    grant(k_event_map, sort) && grant(k_event_finish, finish_smem(kEventPoints));
    if (!ok)
      cudaGetLastError();  // the refusal is not left pending for the next launch
    state = ok ? 1 : -1;
    granted[dev].store(state, std::memory_order_relaxed);
  }
  return state > 0;
}

bool event_path(const RunShape& sh) {
  return sh.n_events == 1 && sh.n >= 1 && sh.n <= kEventPoints && sh.n_tiles <= kEventTiles && clusters_ready();
}

bool event_map_path(int64_t n, int32_t n_clusters) {
  return n >= 1 && n <= kEventPoints && n_clusters <= kEventTiles && clusters_ready();
}

cudaError_t launch_event_front(const RunShape& sh, const RunParams& prm, const RunIO& io, const GridDesc& grid,
                               const EventDesc& ev, const DeviceBuffers& b, cudaStream_t st) {
  FrontArgs a{};
  for (int d = 0; d < sh.D; ++d) {
    a.x[d] = io.coords[d];
    a.sig[d] = io.sigma[d];
  }
  a.weight = io.weight;
  a.unc = io.unc;
  a.tags = io.tags;
  a.grid = grid;
  a.ev = ev;
  a.grids = b.grids;
  a.events = b.events;
  a.point_event = b.point_event;
  a.tile_offset = b.tile_offset;
  a.perm = b.perm;
  a.sevt = b.sorted_event;
  a.sx = b.sorted_coords;
  a.sw = b.sorted_weight;
  a.ssig = b.sorted_sigma;
  a.sunc = b.sorted_unc;
  a.stag = b.sorted_tag;
  static_assert(kEventTiles <= kTileBlocks, "the cell layout of such an event reads records, not coordinate planes");
  a.rec = sweep_fast_path(prm) ? b.rec_dens : nullptr;
  a.event_exact = sh.D == 2 || sh.D == 3 ? b.event_exact : nullptr;
  a.counters = b.counters;
  a.large_count = sweep_fast_path(prm) ? nullptr : b.counters + 3;
  const auto kernel = sh.D == 2 ? k_event_front<2> : sh.D == 3 ? k_event_front<3> : k_event_front<0>;
  return launch_cluster(kernel, cluster_blocks(sh.n), ClusterSort::bytes((int)sh.n_tiles), st, prm, a);
}

cudaError_t launch_event_finish(const RunShape& sh, const RunIO& io, const DeviceBuffers& b, cudaStream_t st) {
  return launch_cluster(k_event_finish, cluster_blocks(sh.n), finish_smem(sh.n), st, (int)sh.n, b.parent, b.perm,
                        b.seed_flag, b.seed_rank, io.cluster_index, b.seeds, b.seed_event, b.counters + 1,
                        b.status, io.host_n_seeds, io.host_status);
}

cudaError_t launch_event_map(int64_t n, const int32_t* labels, int32_t n_clusters, int32_t* offsets,
                             int32_t* points, cudaStream_t st) {
  return launch_cluster(k_event_map, cluster_blocks(n), ClusterSort::bytes(n_clusters), st, (int)n, labels, n_clusters,
                        offsets, points);
}

}  // namespace clue_impl
