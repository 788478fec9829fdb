// validation.cu — cluster centroids and silhouette scores on the device
// (utils/detail/cluster_centroid.hpp:86-140, utils/detail/scores.hpp:24-100).
//
// Both take the cluster -> points map of clue_get_clusters_device (points of
// each cluster in ascending index order, the order the reference's host
// association map holds them) and add in that order with round-to-nearest
// intrinsics, so every centroid and every per-point silhouette is the
// reference's float value bit for bit. Neither allocates.
#include <cfloat>

#include "abi_internal.h"
#include "sweep_device.cuh"

using namespace clue_impl;

namespace clue_impl {

namespace {

struct CoordTable {
  const float* p[kMaxDim];
};

// One block per cluster. Each sum over the cluster's points is a serial chain of
// rounded additions in the map's order, so one lane runs the chain of each
// dimension (and one that of the weights) over 256 points at a time which the
// whole block has gathered (and multiplied by their weights) into shared memory,
// the next 256 being on their way meanwhile. Bound by the additions' latency, not
// by a dependent gather per point as with a thread per (cluster, dimension): 40
// clusters of 740 points took 98 us (weighted 151 us) that way, 12 us (14 us) here.
// (Many clusters: k_centroids_many.)
__global__ void __launch_bounds__(kThreads) k_centroids(int D, CoordTable x, const float* w,
                                                        const int32_t* offsets, const int32_t* members,
                                                        int weighted, float* out) {
  // rows of 257 words: the chains read different banks
  __shared__ float s_v[kMaxDim + 1][kThreads + 1];
  const int64_t c = blockIdx.x;
  const int tid = threadIdx.x;
  const int b = offsets[c], e = offsets[c + 1];
  float sum = 0.0f, next[kMaxDim], next_w = 0.0f;
  auto gather = [&](int k) {  // the point at k + tid of the map
    if (k + tid >= e)
      return;
    const int i = members[k + tid];
    next_w = weighted ? w[i] : 0.0f;
#pragma unroll
    for (int d = 0; d < kMaxDim; ++d)
      if (d < D)
        next[d] = weighted ? __fmul_rn(x.p[d][i], next_w) : x.p[d][i];
  };
  gather(b);
  for (int k = b; k < e; k += kThreads) {
#pragma unroll
    for (int d = 0; d < kMaxDim; ++d)
      if (d < D)
        s_v[d][tid] = next[d];
    s_v[D][tid] = next_w;
    __syncthreads();
    gather(k + kThreads);
    if (tid <= D) {
      const int cnt = min(kThreads, e - k);
#pragma unroll 16
      for (int j = 0; j < cnt; ++j)
        sum = __fadd_rn(sum, s_v[tid][j]);
    }
    __syncthreads();
  }
  if (tid < 32) {
    const float total = __shfl_sync(0xffffffffu, sum, D);
    if (tid < D)
      out[c * D + tid] = weighted ? __fdiv_rn(sum, total) : __fdiv_rn(sum, (float)(e - b));
  }
}

// One thread per (cluster, dimension): from kManyClusters clusters on their chains fill
// the GPU, and a block of 256 threads for each would mostly wait. 2-D, us, a thread / a
// block: 3,000 clusters of 5 points 4.7 / 6.6, of 64 15 / 9; 10,000 of 5 4.7 / 15, of 128
// 27 / 27, in 3-D of 1,024 181 / 258; 100,000 of 5 11 / 103, of 128 140 / 289; 400,000 of
// 32 201 / 759.
constexpr int32_t kManyClusters = 4096;
__global__ void __launch_bounds__(kThreads) k_centroids_many(int D, CoordTable x, const float* w,
                                                             const int32_t* offsets, const int32_t* members,
                                                             int32_t n_clusters, int weighted, float* out) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (int64_t)n_clusters * D)
    return;
  const int c = (int)(t / D), d = (int)(t % D);
  const int b = offsets[c], e = offsets[c + 1];
  float sum = 0.0f, total = 0.0f;
  for (int k = b; k < e; ++k) {
    const int i = members[k];
    const float v = x.p[d][i];
    if (weighted) {
      sum = __fadd_rn(sum, __fmul_rn(v, w[i]));
      total = __fadd_rn(total, w[i]);
    } else {
      sum = __fadd_rn(sum, v);
    }
  }
  out[t] = weighted ? __fdiv_rn(sum, total) : __fdiv_rn(sum, (float)(e - b));
}

__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

// The square root of a number from kRootLow up to FLT_MAX: g = x y from the
// approximate y = 1/sqrt(x), corrected once by the residual x - g^2 of a fused
// multiply-add (Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990): g + (x - g^2) y / 2. That it is the correctly rounded
// root on sm_100 is checked on every float of the range (clue_selftest_math); outside
// it an infinity, a NaN, a subnormal or a zero gives NaN, and another small number may
// be a unit in the last place off. The caller tests the range once for 32 of them.
constexpr float kRootLow = 0x1p-90f;
__device__ __forceinline__ float sqrt_in_range(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  const float g = __fmul_rn(x, y);
  return __fmaf_rn(__fmaf_rn(-g, g, x), __fmul_rn(y, 0.5f), g);
}

// Counts of floats: [0] from kRootLow to FLT_MAX with sqrt_in_range other than __fsqrt_rn,
// [1] from -80 to 0 with clue_expf_normal other than clue_expf, [2] zero, subnormal or
// not finite with a sqrt_in_range that is a number.
__global__ void __launch_bounds__(kThreads) k_math_selftest(unsigned long long* differing) {
  unsigned bad[3] = {0, 0, 0};
  const uint32_t root_low = __float_as_uint(kRootLow), infinite = 0x7f800000u;
  const uint32_t last = __float_as_uint(80.0f) | 0x80000000u;
  for (uint64_t b = (uint64_t)blockIdx.x * kThreads + threadIdx.x; b <= last; b += (uint64_t)gridDim.x * kThreads) {
    const uint32_t bits = (uint32_t)b;
    const float x = __uint_as_float(bits);
    if (bits >= 0x80000000u) {
      bad[1] += __float_as_uint(clue_expf_normal(x)) != __float_as_uint(clue_expf(x));
    } else {
      const float root = sqrt_in_range(x);
      if (bits >= root_low && bits < infinite)
        bad[0] += __float_as_uint(root) != __float_as_uint(__fsqrt_rn(x));
      else if (bits < 0x00800000u || bits >= infinite)
        bad[2] += root == root;
    }
  }
#pragma unroll
  for (int k = 0; k < 3; ++k)
    if (bad[k])
      atomicAdd(&differing[k], (unsigned long long)bad[k]);
}

// Silhouettes: a warp holds 32 points, one per lane, and the sums of distances
// to different clusters do not depend on one another, so the W warps of a group
// share the same 32 points and take the clusters one by one from the group's
// counter. A cluster's points pass through shared memory 32 at a time, the next
// 32 being gathered meanwhile, and every lane adds its distances in the map's
// order. Bound by the issue of the distances: four at a time, the differences and
// squares packed (not their sums: packed products and sums would be contracted),
// the roots by sqrt_in_range. A tile of 32 that is not full, that holds one of the
// lanes' own points, or that gives a squared distance out of that range is taken
// (again) one distance at a time. 32,768 points in 40 clusters: 4.96 ms with one
// thread per point over all clusters, 0.65 ms with __fsqrt_rn, 0.44 ms now.
// DD: the number of dimensions, or 0 for any (D at run time).
template <int DD>
__global__ void __launch_bounds__(kThreads) k_silhouette(int D_any, CoordTable x, const int32_t* labels,
                                                         const int32_t* offsets, const int32_t* members,
                                                         int32_t n_clusters, int64_t n, int W,
                                                         float* scores) {
  constexpr int kDims = DD ? DD : kMaxDim;
  constexpr int kWarps = kThreads / 32;
  const int D = DD ? DD : D_any;
  __shared__ __align__(16) float s_x[kWarps][kDims][32];
  __shared__ int32_t s_m[kWarps][32];
  __shared__ float s_a[kWarps][32], s_b[kWarps][32];
  __shared__ int s_next[kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int group = warp / W;
  const int64_t i = ((int64_t)blockIdx.x * (kWarps / W) + group) * 32 + lane;
  const bool valid = i < n;
  const int own = valid ? labels[i] : -1;
  if (threadIdx.x < kWarps)
    s_next[threadIdx.x] = 0;
  s_a[warp][lane] = 0.0f;
  __syncthreads();
  float xi[kDims];
#pragma unroll
  for (int d = 0; d < kDims; ++d)
    xi[d] = (valid && d < D) ? x.p[d][i] : 0.0f;
  float(*sx)[32] = s_x[warp];
  int32_t* sm = s_m[warp];
  float b = FLT_MAX;
  const auto distance = [&](int j) {
    float dist = 0.0f;
#pragma unroll
    for (int d = 0; d < kDims; ++d)
      if (d < D) {
        const float diff = __fsub_rn(xi[d], sx[d][j]);
        // the sum starts at +0 and a square is never -0: the first addition is exact
        dist = d == 0 ? __fmul_rn(diff, diff) : __fadd_rn(dist, __fmul_rn(diff, diff));
      }
    return __fsqrt_rn(dist);
  };
  for (;;) {
    int c = 0;
    if (lane == 0)
      c = atomicAdd(&s_next[group], 1);
    c = __shfl_sync(0xffffffffu, c, 0);
    if (c >= n_clusters)
      break;
    const int k0 = offsets[c], k1 = offsets[c + 1];
    float sum = 0.0f, next[kDims];
    int next_m = 0;
    auto gather = [&](int k) {
      if (k + lane < k1) {
        next_m = members[k + lane];
#pragma unroll
        for (int d = 0; d < kDims; ++d)
          if (d < D)
            next[d] = x.p[d][next_m];
      }
    };
    gather(k0);
    for (int k = k0; k < k1; k += 32) {
      __syncwarp();  // the previous 32 have been read
      sm[lane] = next_m;
#pragma unroll
      for (int d = 0; d < kDims; ++d)
        if (d < D)
          sx[d][lane] = next[d];
      // whether one of the lanes' own points is among these 32
      const bool mine = __any_sync(0xffffffffu, k + lane < k1 && (next_m >> 5) == (int)(i >> 5));
      __syncwarp();
      if (k + 32 < k1)
        gather(k + 32);
      const int cnt = min(32, k1 - k);
      const float before = sum;
      float least = FLT_MAX;
      const bool whole = cnt == 32 && !mine;
      if (whole) {
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          float2 a, e;
#pragma unroll
          for (int d = 0; d < kDims; ++d)
            if (d < D) {
              const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(&sx[d][j]);
              const unsigned long long own_x = pack2(xi[d], xi[d]);
              const unsigned long long dl = sub2(own_x, v.x), dh = sub2(own_x, v.y);
              const float2 sl = unpack2(mul2(dl, dl)), sh = unpack2(mul2(dh, dh));
              a = d == 0 ? sl : make_float2(__fadd_rn(a.x, sl.x), __fadd_rn(a.y, sl.y));
              e = d == 0 ? sh : make_float2(__fadd_rn(e.x, sh.x), __fadd_rn(e.y, sh.y));
            }
          least = fminf(fminf(least, fminf(a.x, a.y)), fminf(e.x, e.y));
          sum = __fadd_rn(__fadd_rn(sum, sqrt_in_range(a.x)), sqrt_in_range(a.y));
          sum = __fadd_rn(__fadd_rn(sum, sqrt_in_range(e.x)), sqrt_in_range(e.y));
        }
      }
      // not (whole and in range): a zero or an infinity gave NaN
      if (!whole || !(least >= kRootLow) || sum != sum) {
        sum = before;
        for (int j = 0; j < cnt; ++j) {
          const float dist = distance(j);
          if (sm[j] != (int)i)
            sum = __fadd_rn(sum, dist);
        }
      }
    }
    if (own == c) {
      s_a[group * W][lane] = __fdiv_rn(sum, (float)(k1 - k0 - 1));
    } else {
      const float mean = __fdiv_rn(sum, (float)(k1 - k0));  // an empty cluster's NaN is not smaller
      b = mean < b ? mean : b;                              // std::min(acc, val)
    }
  }
  s_b[warp][lane] = b;
  __syncthreads();
  if (warp % W == 0 && valid) {
    const float a = s_a[warp][lane];
    for (int r = 1; r < W; ++r)
      b = s_b[warp + r][lane] < b ? s_b[warp + r][lane] : b;
    const bool take = own >= 0 && own < n_clusters && offsets[own + 1] - offsets[own] >= 2;
    const float hi = a < b ? b : a;  // std::max(a, b)
    scores[i] = take ? __fdiv_rn(__fsub_rn(b, a), hi) : __int_as_float(0x7fc00000);
  }
}

// Warps that share a group's points: as many as there are clusters to share, up
// to 8, while the groups alone leave the GPU room (128 warps for each SM in all, 32
// of which run at once, so that the last wave is not mostly empty). Blocks of 4 warps
// and groups all resident at once measured slower: their warps are too few to hide
// the chains of additions (65,536 points: 2,265 us against 1,830 a call).
int silhouette_split(int64_t n, int32_t n_clusters) {
  const int64_t groups = (n + 31) / 32;
  int W = 1;
  while (W < kThreads / 32 && 2 * W <= n_clusters && groups * 2 * W <= (int64_t)sm_count() * 128)
    W *= 2;
  return W;
}

clue_status check_map(const clue_points* pts, const int32_t* offsets, const int32_t* members,
                      int32_t n_clusters) {
  if (!pts || pts->ndim < 1 || pts->ndim > kMaxDim || pts->n <= 0)
    return fail(CLUE_ERR_INVALID_ARGUMENT, "points with 1..10 dimensions and n > 0 are required");
  for (int d = 0; d < pts->ndim; ++d)
    if (!pts->coords[d])
      return fail(CLUE_ERR_INVALID_ARGUMENT, "a coordinate plane is null");
  if (n_clusters < 0 || (n_clusters > 0 && (!offsets || !members)))
    return fail(CLUE_ERR_INVALID_ARGUMENT, "the cluster map is required");
  return CLUE_OK;
}

}  // namespace

}  // namespace clue_impl

extern "C" {

clue_status clue_cluster_centroids_device(const clue_points* points, const int32_t* cluster_offsets,
                                          const int32_t* cluster_points, int32_t n_clusters,
                                          int32_t weighted, float* centroids, void* stream) {
  clue_status s = check_map(points, cluster_offsets, cluster_points, n_clusters);
  if (s != CLUE_OK)
    return s;
  if (weighted && !points->weight)
    return fail(CLUE_ERR_INVALID_ARGUMENT, "weighted centroids need the weights");
  if (n_clusters == 0)
    return CLUE_OK;
  if (!centroids)
    return fail(CLUE_ERR_INVALID_ARGUMENT, "the centroid output is required");
  CoordTable x{};
  for (int d = 0; d < points->ndim; ++d)
    x.p[d] = points->coords[d];
  const cudaStream_t st = (cudaStream_t)stream;
  if (n_clusters < kManyClusters) {
    k_centroids<<<n_clusters, kThreads, 0, st>>>(points->ndim, x, points->weight, cluster_offsets, cluster_points,
                                                 weighted ? 1 : 0, centroids);
  } else {
    const int64_t threads = (int64_t)n_clusters * points->ndim;
    k_centroids_many<<<(int)((threads + kThreads - 1) / kThreads), kThreads, 0, st>>>(
        points->ndim, x, points->weight, cluster_offsets, cluster_points, n_clusters, weighted ? 1 : 0, centroids);
  }
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? CLUE_OK : fail_cuda(e, "centroid kernel launch");
}

clue_status clue_silhouette_device(const clue_points* points, const int32_t* cluster_offsets,
                                   const int32_t* cluster_points, int32_t n_clusters, float* scores,
                                   void* stream) {
  clue_status s = check_map(points, cluster_offsets, cluster_points, n_clusters);
  if (s != CLUE_OK)
    return s;
  if (!points->cluster_index || !scores)
    return fail(CLUE_ERR_INVALID_ARGUMENT, "labels (cluster_index) and the score output are required");
  CoordTable x{};
  for (int d = 0; d < points->ndim; ++d)
    x.p[d] = points->coords[d];
  const int W = silhouette_split(points->n, n_clusters);
  const int per_block = kThreads / W;  // points
  const int blocks = (int)(((int64_t)points->n + per_block - 1) / per_block);
  const auto launch = [&](auto kernel) {
    kernel<<<blocks, kThreads, 0, (cudaStream_t)stream>>>(points->ndim, x, points->cluster_index, cluster_offsets,
                                                          cluster_points, n_clusters, points->n, W, scores);
  };
  switch (points->ndim) {
    case 1: launch(k_silhouette<1>); break;
    case 2: launch(k_silhouette<2>); break;
    case 3: launch(k_silhouette<3>); break;
    default: launch(k_silhouette<0>); break;
  }
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? CLUE_OK : fail_cuda(e, "silhouette kernel launch");
}

clue_status clue_selftest_math(int32_t device, void* stream, int64_t* differing) {
  if (!differing)
    return fail(CLUE_ERR_INVALID_ARGUMENT, "the counts are required");
  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess)
    return fail_cuda(e, "cudaSetDevice");
  constexpr size_t kBytes = 3 * sizeof(unsigned long long);
  unsigned long long* counts = nullptr;
  if ((e = cudaMalloc(&counts, kBytes)) != cudaSuccess)
    return fail_cuda(e, "self-test allocation");
  const cudaStream_t st = (cudaStream_t)stream;
  if ((e = cudaMemsetAsync(counts, 0, kBytes, st)) == cudaSuccess) {
    k_math_selftest<<<sm_count() * 16, kThreads, 0, st>>>(counts);
    if ((e = cudaGetLastError()) == cudaSuccess &&
        (e = cudaMemcpyAsync(differing, counts, kBytes, cudaMemcpyDeviceToHost, st)) == cudaSuccess)
      e = cudaStreamSynchronize(st);
  }
  cudaFree(counts);
  return e == cudaSuccess ? CLUE_OK : fail_cuda(e, "math self-test");
}

}  // extern "C"
