// sweep_device.cuh — device building blocks shared by the sweep kernels: search
// boxes and tiles, packed squared distances, and the cell layout.
#pragma once

#include <cfloat>

#include "sweep.cuh"

namespace clue_impl {

namespace {

constexpr int kThreads = 256;
constexpr unsigned kFullMask = 0xffffffffu;
// sqrtf(2.0f), correctly rounded (the reference's math::sqrt(TData{2})).
constexpr float kSqrt2 = 1.41421356237309504880f;

// Search box of point s: bins [inf, sup] per dimension (TilesView.hpp:77-87),
// half width max(r, r * sigma * sqrt(2)) (ClusteringKernels.hpp:112-118).
template <int D>
__device__ __forceinline__ void search_box(const GridDesc& g, const RunParams& p, const float* xi,
                                           const float* si, float radius, int* inf, int* sup) {
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const float r = std_max(radius, __fmul_rn(__fmul_rn(radius, si[d]), kSqrt2));
    inf[d] = get_bin(g, p, __fsub_rn(xi[d], r), d);
    sup[d] = get_bin(g, p, __fadd_rn(xi[d], r), d);
    if (p.wrapped[d] && inf[d] > sup[d])
      sup[d] += g.k;
  }
}

// Advances the tile odometer (last dimension fastest); false when exhausted.
template <int D>
__device__ __forceinline__ bool next_tile(int* b, const int* inf, const int* sup) {
  bool carry = true;
#pragma unroll
  for (int d = D - 1; d >= 0; --d) {
    if (carry) {
      if (b[d] < sup[d]) {
        ++b[d];
        carry = false;
      } else {
        b[d] = inf[d];
      }
    }
  }
  return !carry;
}

template <int D>
__device__ __forceinline__ int tile_id(const GridDesc& g, const RunParams& p, int base, const int* b) {
  int t = base;
#pragma unroll
  for (int d = 0; d < D; ++d)
    t += g.stride[d] * wrap_bin(g, p, b[d], d);
  return t;
}

template <int D>
__device__ __forceinline__ void load_point(const RunParams& p, const SweepArgs& a, int64_t s, float* x,
                                           float* sg) {
#pragma unroll
  for (int d = 0; d < D; ++d) {
    x[d] = a.sx[d * a.n + s];
    sg[d] = ((p.has_sigma >> d) & 1) ? a.ssig[d * a.n + s] : 0.0f;
  }
}

constexpr int kAnyMetric = -1;  // the metric of the run, decided per pair

// metric_inner for the metric of the instantiation.
template <int D, int METRIC>
__device__ __forceinline__ float inner_distance(const RunParams& p, const float* xi, const float* xj, const float* si,
                                                const float* sj) {
  if (METRIC == kAnyMetric)
    return metric_inner<D>(p, xi, xj, si, sj);
  float acc = 0.0f;
#pragma unroll
  for (int d = D - 1; d >= 0; --d) {
    float diff = __fsub_rn(xi[d], xj[d]);
    if (METRIC == CLUE_METRIC_PERIODIC_EUCLIDEAN) {
      diff = fabsf(diff);
      diff = std_min(diff, __fsub_rn(p.mparam[d], diff));
    }
    // the right fold starts from +0 and a square is never -0: exact
    acc = d == D - 1 ? __fmul_rn(diff, diff) : __fadd_rn(__fmul_rn(diff, diff), acc);
  }
  return acc;
}

// Order-preserving image of a density: key(a) > key(b) iff a > b and equal
// densities give equal keys. NaN maps to 0, below every number, so a NaN
// density is never "higher" (every comparison with NaN is false). Densities
// are never -0 (they start at +0 and round-to-nearest sums of opposite values
// give +0), so no other pair of equal values has different keys.
__device__ __forceinline__ uint32_t rho_key(float rho) {
  if (rho != rho)
    return 0u;
  const uint32_t b = __float_as_uint(rho);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// (x_i - x_j)^2 and (y_i - y_j)^2 with one packed subtract and one packed
// multiply (sm_100 f32x2): each half is the IEEE round-to-nearest result of
// the scalar operation, so the values equal __fsub_rn / __fmul_rn.
__device__ __forceinline__ void sq_diff_xy(float xi, float yi, float xj, float yj, float& sx,
                                           float& sy) {
  asm("{\n\t.reg .b64 a, b, d, s;\n\t"
      "mov.b64 a, {%2, %3};\n\t"
      "mov.b64 b, {%4, %5};\n\t"
      "sub.rn.f32x2 d, a, b;\n\t"
      "mul.rn.f32x2 s, d, d;\n\t"
      "mov.b64 {%0, %1}, s;\n\t}"
      : "=f"(sx), "=f"(sy)
      : "f"(xi), "f"(yi), "f"(xj), "f"(yj));
}

template <int D>
__device__ __forceinline__ float sq_dist(const float* xi, const float4& r) {
  // meta::accumulate right fold: dx^2 + (dy^2 [+ dz^2])
  float sx, sy;
  sq_diff_xy(xi[0], xi[1], r.x, r.y, sx, sy);
  if (D == 2)
    return __fadd_rn(sx, sy);
  const float dz = __fsub_rn(xi[2], r.z);
  return __fadd_rn(sx, __fadd_rn(sy, __fmul_rn(dz, dz)));
}

// ---------------------------------------------------------------------------
// Cell layout (fast path).
//
// Every tile of m points is split into s^D cells, s the largest value with
// s^D * kCellTarget <= m (at least 1, at most cell_dim_max). A point's cell
// comes from cell_coord, which is monotone in the coordinate; a search
// therefore finds every point of [a, b] in the cells cell_coord(a) ..
// cell_coord(b), whatever rounding placed it there. Each cell records the
// bounding box of its members and (for the nearest-higher search) their
// largest key. The density sweep uses the cells to skip candidates no lane of
// a warp can reach; the nearest-higher search visits them nearest-first.
// ---------------------------------------------------------------------------

// Cell coordinate of x in a tile with origin lo and inverse cell width inv
// (0 for a degenerate tile): monotone non-decreasing in x for every non-NaN x,
// clamped to [0, s); NaN lands in cell 0.
__device__ __forceinline__ int cell_coord(float x, float lo, float inv, int s) {
  float u = __fmul_rn(__fsub_rn(x, lo), inv);
  u = fminf(fmaxf(u, 0.0f), (float)(s - 1));
  return (int)u;
}

template <int D>
__device__ __forceinline__ void load_geom(const SweepArgs& a, int t, float* lo, float* inv) {
  const float4 g0 = a.cell_geom[D == 2 ? t : 2 * t];
  if (D == 2) {
    lo[0] = g0.x, lo[1] = g0.y, inv[0] = g0.z, inv[1] = g0.w;
  } else {
    const float4 g1 = a.cell_geom[2 * t + 1];
    lo[0] = g0.x, lo[1] = g0.y, lo[D - 1] = g0.z, inv[0] = g0.w, inv[1] = g1.x, inv[D - 1] = g1.y;
  }
}

template <int D>
__device__ __forceinline__ void load_box(const SweepArgs& a, int slot, float* mn, float* mx) {
  const float4 b0 = a.cell_box[D == 2 ? slot : 2 * slot];
  if (D == 2) {
    mn[0] = b0.x, mn[1] = b0.y, mx[0] = b0.z, mx[1] = b0.w;
  } else {
    const float4 b1 = a.cell_box[2 * slot + 1];
    mn[0] = b0.x, mn[1] = b0.y, mn[D - 1] = b0.z, mx[0] = b0.w, mx[1] = b1.x, mx[D - 1] = b1.y;
  }
}

// Lower bound of the squared distance from xi to any member of a cell, with
// the operations of sq_dist: per dimension the gap to the box is at most
// |fl(x_i - x_j)| of every member (rounding is monotone), and squares and the
// right fold are monotone too.
template <int D>
__device__ __forceinline__ float box_lower_bound(const float* xi, const float* mn, const float* mx) {
  float gap[D];
#pragma unroll
  for (int d = 0; d < D; ++d)
    gap[d] = fmaxf(fmaxf(__fsub_rn(mn[d], xi[d]), __fsub_rn(xi[d], mx[d])), 0.0f);
  if (D == 2)
    return __fadd_rn(__fmul_rn(gap[0], gap[0]), __fmul_rn(gap[1], gap[1]));
  return __fadd_rn(__fmul_rn(gap[0], gap[0]),
                   __fadd_rn(__fmul_rn(gap[1], gap[1]), __fmul_rn(gap[D - 1], gap[D - 1])));
}

// |x_j - x_i| <= reach(bound2) in every coordinate for every point with
// fl(d2) <= bound2: each square and sum is rounded to nearest, so
// |x_j - x_i| <= sqrt(bound2) (1 + 2^-22); the factor 1 + 10^-6 and the
// absolute 10^-19 (square roots near the smallest normal) cover that, rounded up.
__device__ __forceinline__ float reach(float bound2) {
  return __fadd_ru(__fmul_ru(__fsqrt_ru(bound2), 1.000001f), 1e-19f);
}

// Distance from the interval [x_lo, x_hi] to the slab of cell c along one dimension,
// less a margin that covers the rounding of cell_coord and of the slab's ends. The
// first and last cells also hold what lies beyond them.
__device__ __forceinline__ float slab_gap(float x_lo, float x_hi, int c, int s, float lo, float inv) {
  if (!(inv > 0.0f))
    return 0.0f;
  const float width = __fdividef(1.0f, inv);
  const float margin = 1e-5f * (fabsf(lo) + (float)s * width);
  const float below = lo + (float)c * width - x_hi, above = x_lo - (lo + (float)(c + 1) * width);
  const float gap = fmaxf(c > 0 ? below : 0.0f, c < s - 1 ? above : 0.0f);
  return fmaxf(gap - margin, 0.0f);
}

// Asynchronous 16-byte global -> shared copies (per thread, completion by
// commit groups).
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// (a, b) as one 64-bit register pair, the operand of the f32x2 instructions.
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}

// Squared distance and contribution weight of a streamed record: xi_xy holds
// (x_i, y_i) packed, the record arrives as two packed halves {(x, y), (z or v,
// v or w)}; the arithmetic is that of sq_dist.
template <int D>
__device__ __forceinline__ float packed_d2(unsigned long long xi_xy, float zi, const ulonglong2& r,
                                           float& v) {
  float sx, sy;
  asm("{\n\t.reg .b64 d, s;\n\t"
      "sub.rn.f32x2 d, %2, %3;\n\t"
      "mul.rn.f32x2 s, d, d;\n\t"
      "mov.b64 {%0, %1}, s;\n\t}"
      : "=f"(sx), "=f"(sy)
      : "l"(xi_xy), "l"(r.x));
  float hi_lo, hi_hi;  // the record's second half: D = 2 {v, w}; D = 3 {z, v}
  asm("mov.b64 {%0, %1}, %2;" : "=f"(hi_lo), "=f"(hi_hi) : "l"(r.y));
  v = D == 2 ? hi_lo : hi_hi;
  if (D == 2)
    return __fadd_rn(sx, sy);
  const float dz = __fsub_rn(zi, hi_lo);
  return __fadd_rn(sx, __fadd_rn(sy, __fmul_rn(dz, dz)));
}

}  // namespace

}  // namespace clue_impl
