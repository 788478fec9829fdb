// density_group.cu — local density (core/detail/ClusteringKernels.hpp:29-140) with
// G lanes per point, on the fast path (2-D or 3-D, Euclidean, no sigma, no wrapped
// coordinate).
//
// The lanes of a group find the rows of cells within reach of their point, in the
// tiles of its search box, G tiles and then G rows at a time, and test the members
// of a row together. An event whose sums are exact in any order
// (event_sums_exact) adds the hits as they come. Otherwise the reference's order
// decides the roundings: tile by tile, a tile's points in ascending index, i.e.
// ascending sorted position, which the cells permute. The hits are then marked in a
// bitmap over the sorted positions of the tiles; expanded, it gives them in order,
// G at a time: every lane evaluates one contribution and the group adds them one
// after another.
// A point has only its own candidates here, where a warp of 32 points (k_density_fast)
// tests those of all of them: points far apart (noise) cost little, and small runs
// spread over the GPU. Bound by latency (37 % of the warp slots active, issue on 48 %
// of the cycles at 65,536 points) and by what a group of lanes spends on tiles and
// rows before its first test, so larger runs keep 32 points per warp. Density, us,
// 32 points per warp / 32 lanes / 16 lanes per point: 2-D events of 1,024 points
// 35 / 20 / 31, 8,192: 82 / 29 / 35, 16,384: 98 / 43 / 41, 49,152: 149 / 109 / 98,
// 65,536: 131 / 137 / 125, 131,072: 181 / 283 / 260; with the Gaussian kernel 8,192:
// 406 / 53 / 74, 16,384: 348 / 86 / 86; 3-D showers 1,024: 31 / 12 / 12, 16,384: 121 /
// 47 / 41, 65,536: 359 / 248 / 229. (8 lanes per point lost to 16 up to 16,384.)
// (Measured with 7 blocks per SM; 16 lanes in 2-D are 5 to 9 % faster now, see launch.)
// Those are blobs and showers of a few hundred candidates per point. Crowded tiles make
// the lanes lose, so the cell layout estimates both forms (density_by_load, add_load).
// The warp stays converged: groups that are done wait for the others, and every
// shuffle and vote is reached by all 32 lanes.
#include <climits>

#include "engine.h"
#include "sweep_device.cuh"

namespace clue_impl {

namespace {

// One tile of a point's search box.
struct NearTile {
  int row;       // rows in reach of the group's earlier tiles
  int bit;       // points of the group's earlier tiles
  int begin;     // first sorted position, also the first slot of its cells
  int points;
  int s;         // cells per dimension
  int c0, c1;    // first cell in reach in dimensions 0 and 1
  int n1;        // cells in reach along dimension 1 (3-D)
  float lo[3], inv[3];
};

template <int G>
struct NearGroup {
  static constexpr int kWords = 128;  // bitmap of 4,096 sorted positions
  static constexpr int kBits = 32 * kWords;
  NearTile tile[G];
  int row_off[G];    // members of the rows before each of G rows
  int row_first[G];  // its first member, less row_off
  int row_bit[G];    // from a member's sorted position to its bit
  __align__(16) float add[G];  // contributions, in order
  uint32_t bitmap[kWords];
  uint16_t list[32 * G];  // the set bits of G words, in order
};

template <int D, int KIND, bool NORMAL, int G, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_density_group(const RunParams p, const SweepArgs a) {
  constexpr int P = 32 / G;  // points of a warp at a time
  constexpr int kBits = NearGroup<G>::kBits;
  extern __shared__ __align__(16) unsigned char s_dyn[];
  const int64_t n = a.n;
  const int lane = threadIdx.x & 31, l = lane % G, g0 = lane - l;
  NearGroup<G>& sh = reinterpret_cast<NearGroup<G>*>(s_dyn)[threadIdx.x / G];
  const float4* __restrict__ rec = a.rec_dens;
  const float4* __restrict__ rec_cell = a.rec_cell;
  const float R = reach(p.dc2);
  const float R2 = __fmul_ru(R, R);
  if (G < 32 && density_streams<D>(a))
    return;
  for (;;) {
    int64_t w0 = 0;
    if (lane == 0)
      w0 = atomicAdd(reinterpret_cast<unsigned*>(&a.queue[0]), (unsigned)P);
    w0 = __shfl_sync(kFullMask, w0, 0);
    if (w0 >= n)
      break;
    const int64_t w = w0 + lane / G;
    // groups past the end shadow the warp's first point and write nothing
    const bool active = w < n;
    const int64_t at = active ? w : w0;
    const int s = a.work_dens ? a.work_dens[at] : a.nh_q[at];  // neighbours follow one another
    const int event = a.sevt[s];
    const EventDesc ev = a.events[event];
    const GridDesc& g = a.grids[ev.grid];
    const float4 ri = rec[s];
    const float xi[3] = {ri.x, ri.y, ri.z};
    const float zero[3] = {0.0f, 0.0f, 0.0f};
    const float wi = a.sw[s];
    int inf[D], sup[D];
    search_box<D>(g, p, xi, zero, p.dc, inf, sup);
    bool self_in = true;  // the own tile is in the box and the point in range of itself
    int64_t box = 1;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const int own = get_bin(g, p, xi[d], d);
      self_in &= inf[d] <= own && own <= sup[d] && isfinite(xi[d]);
      box *= max(sup[d] - inf[d] + 1, 0);
    }
    const bool exact = KIND == CLUE_KERNEL_FLAT && event_sums_exact(a.event_exact, event, ev.n);
    const bool some_ordered = __any_sync(kFullMask, !exact);
    float rho = 0.0f;
    int tested = 0;
    for (int64_t tb = 0; __any_sync(kFullMask, tb < box); tb += G) {
      // ---- the box's next G tiles, one per lane ----
      int rows = 0, m = 0;
      NearTile nt;
      nt.begin = nt.points = 0, nt.s = 1, nt.c0 = nt.c1 = 0, nt.n1 = 1;
#pragma unroll
      for (int d = 0; d < 3; ++d)
        nt.lo[d] = nt.inv[d] = 0.0f;
      if (tb + l < box) {
        int b[D];
        int64_t rem = tb + l;  // (boxes of fewer than 2^31 tiles: tile ids are 32-bit)
#pragma unroll
        for (int d = D - 1; d > 0; --d) {
          const unsigned nd = (unsigned)(sup[d] - inf[d] + 1);
          const unsigned q = (unsigned)rem / nd;
          b[d] = inf[d] + (int)((unsigned)rem - q * nd);
          rem = q;
        }
        b[0] = inf[0] + (int)rem;
        int t = ev.tile_base;
#pragma unroll
        for (int d = 0; d < D; ++d)
          t += g.stride[d] * b[d];
        nt.begin = a.tile_offset[t];
        m = nt.points = a.tile_offset[t + 1] - nt.begin;
        if (m > 0) {
          nt.s = a.cell_s[t];
          load_geom<D>(a, t, nt.lo, nt.inv);
          int lo[D], hi[D];
#pragma unroll
          for (int d = 0; d < D; ++d) {
            lo[d] = cell_coord(__fsub_rd(xi[d], R), nt.lo[d], nt.inv[d], nt.s);
            hi[d] = cell_coord(__fadd_ru(xi[d], R), nt.lo[d], nt.inv[d], nt.s);
          }
          nt.c0 = lo[0];
          rows = hi[0] - lo[0] + 1;
          if (D == 3) {
            nt.c1 = lo[1];
            nt.n1 = hi[1] - lo[1] + 1;
            rows *= nt.n1;
          }
        }
      }
      int row_end = rows, bit_end = m;
#pragma unroll
      for (int o = 1; o < G; o <<= 1) {
        const int y0 = __shfl_up_sync(kFullMask, row_end, o), y1 = __shfl_up_sync(kFullMask, bit_end, o);
        if (l >= o) {
          row_end += y0;
          bit_end += y1;
        }
      }
      const int n_rows = __shfl_sync(kFullMask, row_end, g0 + G - 1);
      const int all_bits = __shfl_sync(kFullMask, bit_end, g0 + G - 1);
      const int n_bits = exact ? 1 : all_bits;
      nt.row = row_end - rows;
      nt.bit = bit_end - m;
      __syncwarp();
      sh.tile[l] = nt;
      __syncwarp();
      // ---- the tiles' points, a bitmap's worth at a time (exact sums: at once) ----
      for (int b0 = 0; __any_sync(kFullMask, b0 < n_bits); b0 += kBits) {
        const bool window = b0 < n_bits;
        if (some_ordered) {
          for (int k = l; k < NearGroup<G>::kWords && k * 32 < all_bits; k += G)
            sh.bitmap[k] = 0;
          __syncwarp();
        }
        for (int f0 = 0; __any_sync(kFullMask, window && f0 < n_rows); f0 += G) {
          // ---- one row of cells per lane ----
          const int f = f0 + l;
          int start = 0, end = 0, shift = 0;
          if (window && f < n_rows) {
            int t = 0;  // the last tile whose rows start at or before f
#pragma unroll
            for (int o = G / 2; o > 0; o >>= 1)
              if (sh.tile[t + o].row <= f)
                t += o;
            const NearTile& ct = sh.tile[t];
            shift = ct.bit - ct.begin - b0;
            int r = f - ct.row, c1 = 0;
            if (D == 3) {
              // quotient of integers below 2^8: far from the rounding
              const int q = (int)__fdividef((float)r + 0.5f, (float)ct.n1);
              c1 = ct.c1 + r - q * ct.n1;
              r = q;
            }
            const int c0 = ct.c0 + r;
            // what is left of the reach along the last dimension
            const float gap0 = slab_gap(xi[0], xi[0], c0, ct.s, ct.lo[0], ct.inv[0]);
            const float gap1 = D == 3 ? slab_gap(xi[1], xi[1], c1, ct.s, ct.lo[1], ct.inv[1]) : 0.0f;
            const float left2 = R2 * 1.00001f - gap0 * gap0 - gap1 * gap1;
            // (a NaN coordinate has no gap and no cells but the first)
            const bool here = exact || (ct.bit < b0 + kBits && ct.bit + ct.points > b0);
            if (here && !(left2 < 0.0f)) {
              const float left = fminf(__fsqrt_ru(left2) * 1.00001f, R);
              const int lo = cell_coord(__fsub_rd(xi[D - 1], left), ct.lo[D - 1], ct.inv[D - 1], ct.s);
              const int hi = cell_coord(__fadd_ru(xi[D - 1], left), ct.lo[D - 1], ct.inv[D - 1], ct.s);
              const CellInfo* info = a.cell_info + ct.begin + (D == 2 ? c0 * ct.s : (c0 * ct.s + c1) * ct.s);
              start = info[lo].start;
              end = info[hi].end;
            }
          }
          // ---- the rows' members, dealt to the lanes, kAhead loads in flight ----
          const int len = max(end - start, 0);
          int off = len;
#pragma unroll
          for (int o = 1; o < G; o <<= 1) {
            const int y = __shfl_up_sync(kFullMask, off, o);
            if (l >= o)
              off += y;
          }
          const int total = __shfl_sync(kFullMask, off, g0 + G - 1);
          off -= len;
          __syncwarp();
          sh.row_off[l] = off;
          sh.row_first[l] = start - off;
          sh.row_bit[l] = shift;
          __syncwarp();
          tested += total;
          constexpr int kAhead = 4;
          for (int m0 = 0; __any_sync(kFullMask, m0 < total); m0 += kAhead * G) {
            float4 r[kAhead];
            int q[kAhead], to_bit[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
              const int k = m0 + u * G + l;
              q[u] = -1;
              if (k < total) {
                int row = 0;  // the last row whose members start at or before k
#pragma unroll
                for (int o = G / 2; o > 0; o >>= 1)
                  if (sh.row_off[row + o] <= k)
                    row += o;
                q[u] = sh.row_first[row] + k;
                to_bit[u] = sh.row_bit[row];
                r[u] = __ldg(&rec_cell[q[u]]);
              }
            }
#pragma unroll
            for (int u = 0; u < kAhead; ++u)
              if (q[u] >= 0 && sq_dist<D>(xi, r[u]) <= p.dc2) {
                if (exact) {
                  rho = __fadd_rn(rho, D == 2 ? r[u].z : r[u].w);
                } else {
                  const int bit = a.nh_q[q[u]] + to_bit[u];
                  if ((unsigned)bit < (unsigned)kBits)
                    atomicOr(&sh.bitmap[bit >> 5], 1u << (bit & 31));
                }
              }
          }
          __syncwarp();
        }
        if (!some_ordered)
          continue;
        // ---- ordered sums: the bitmap's set bits, in order, G words at a time ----
        const int words = exact || !window ? 0 : (min(all_bits - b0, kBits) + 31) / 32;
        for (int k0 = 0; __any_sync(kFullMask, k0 < words); k0 += G) {
          const uint32_t word = k0 + l < words ? sh.bitmap[k0 + l] : 0u;
          if (!__any_sync(kFullMask, word != 0))
            continue;
          int at = __popc(word);
#pragma unroll
          for (int o = 1; o < G; o <<= 1) {
            const int y = __shfl_up_sync(kFullMask, at, o);
            if (l >= o)
              at += y;
          }
          const int hits = __shfl_sync(kFullMask, at, g0 + G - 1);
          at -= __popc(word);
          for (uint32_t bits = word; bits; bits &= bits - 1)
            sh.list[at++] = (uint16_t)((k0 + l) * 32 + __ffs(bits) - 1);
          __syncwarp();
          for (int h = 0; __any_sync(kFullMask, h < hits); h += G) {
            float add = 0.0f;  // (a sum is never -0, so adding +0 leaves it)
            if (h + l < hits) {
              const int bit = b0 + sh.list[h + l];
              int t = 0;  // the last tile whose points start at or before the bit
#pragma unroll
              for (int o = G / 2; o > 0; o >>= 1)
                if (sh.tile[t + o].bit <= bit)
                  t += o;
              const int q = sh.tile[t].begin + bit - sh.tile[t].bit;
              const float4 r = __ldg(&rec[q]);
              const float v = D == 2 ? r.z : r.w;
              if (KIND == CLUE_KERNEL_FLAT)
                add = q == s ? wi : v;
              else
                add = __fmul_rn(kernel_value_of<KIND, NORMAL>(p, __fsqrt_rn(sq_dist<D>(xi, r)), q == s), v);
            }
            sh.add[l] = add;
            __syncwarp();
#pragma unroll
            for (int j = 0; j < G; j += 4) {
              const float4 v = *reinterpret_cast<const float4*>(&sh.add[j]);
              rho = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(rho, v.x), v.y), v.z), v.w);
            }
            __syncwarp();
          }
          __syncwarp();  // the list is rewritten
        }
      }
    }
    if (KIND == CLUE_KERNEL_FLAT) {
      // the lanes' shares of an exact sum, and the own term: the own record (d2 =
      // 0, in range) added v_i = fl(flat * w_i) where the reference adds w_i. Every
      // step is exact (multiples of u, between 0 and the event bound).
      float sum = rho;
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1)
        sum = __fadd_rn(sum, __shfl_xor_sync(kFullMask, sum, o));
      if (exact)
        rho = self_in ? __fadd_rn(__fsub_rn(sum, __fmul_rn(p.kernel_p0, wi)), wi) : sum;
    }
    if (a.stats) {  // warp-uniform
      const int sum = __reduce_add_sync(kFullMask, active && l == 0 ? tested : 0);
      if (lane == 0) {
        atomicAdd(&a.stats[0], (unsigned long long)sum);
        if (w0 % 32 == 0)
          atomicAdd(&a.stats[1], 1ull);
      }
    }
    if (!active || l != 0)
      continue;
    a.srho[s] = rho;
    const int gi = a.perm[s];
    if (a.out_rho)
      a.out_rho[gi] = rho;
    const uint32_t tag = p.has_tags ? a.stag[s] : (uint32_t)gi;
    const uint32_t kbits = rho_key(rho);
    const int pos = a.nh_pos[s];
    atomicMax(&a.cell_info[a.cell_slot[s]].maxkey, ((unsigned long long)kbits << 32) | tag);
    if (D == 2) {
      a.rec_nh[pos] = make_float4(xi[0], xi[1], __uint_as_float(kbits), __uint_as_float(tag));
    } else {
      a.rec_nh[pos] = make_float4(xi[0], xi[1], xi[2], __uint_as_float(kbits));
      a.rec_tag[pos] = tag;
    }
  }
}

template <int D, int KIND, bool NORMAL, int G>
cudaError_t launch(const RunParams& p, const SweepArgs& a, cudaStream_t st) {
  constexpr int NT = 128;
  constexpr int smem = (int)sizeof(NearGroup<G>) * (NT / G);
  const int64_t blocks = (a.n * G + NT - 1) / NT;
  // Blocks per SM: in 2-D 9 (56 registers) took 39 and 90 us of 16,384 and 50,021
  // points against 41 and 99 with 7, and 44 and 100 with 10; in 3-D 7
  // took 27 us of 10,000 points and 225 of 65,536 against 33 and 252 with 9.
  constexpr int kMinBlocks = D == 2 ? 9 : 7;
  const auto kernel = k_density_group<D, KIND, NORMAL, G, NT, kMinBlocks>;
  kernel<<<(int)std::max<int64_t>(1, std::min<int64_t>(blocks, (int64_t)sm_count() * 16)), NT, smem, st>>>(p, a);
  count_launches(1);
  return cudaGetLastError();
}

template <int D, int G>
cudaError_t launch_kind(const RunParams& p, const SweepArgs& a, cudaStream_t st) {
  switch (p.kernel_kind) {
    case CLUE_KERNEL_FLAT: return launch<D, CLUE_KERNEL_FLAT, false, G>(p, a, st);
    case CLUE_KERNEL_GAUSSIAN:
      return kernel_value_normal(p) ? launch<D, CLUE_KERNEL_GAUSSIAN, true, G>(p, a, st)
                                    : launch<D, CLUE_KERNEL_GAUSSIAN, false, G>(p, a, st);
    default:
      return kernel_value_normal(p) ? launch<D, CLUE_KERNEL_EXPONENTIAL, true, G>(p, a, st)
                                    : launch<D, CLUE_KERNEL_EXPONENTIAL, false, G>(p, a, st);
  }
}

}  // namespace

// From kGroupWide points on a tile can fill several windows of the bitmap, and the flat
// kernel's ordered sums, which a group adds one hit after another, can lose to 32 points
// per warp; the smooth kernels, which those evaluate for all their points, can where n x
// windows is above 46,000. Below, one launch is the better: the second takes 3 us.
// Density, us, lanes per point / 32 points per warp, 65,536 points: ordered flat sums of
// 2-D blobs of 800 points 250 / 138, of 6,400 1,645 / 482, of 16,384 9,554 / 1,435, in 3-D
// of 1,600 344 / 237; Gaussian of 16,384 8,724 / 3,309 and of 6,400 1,602 / 1,950 (lanes
// taken), in 3-D 8,663 / 1,834; exact sums in 3-D of 6,400 479 / 353, but in 2-D 448 / 469
// (lanes taken). All points in one cell (an outlier at 10,000 times the extent), whole
// call: 176 ms / 12.5 ms.
bool density_by_load(const RunParams& p, int64_t n, int32_t n_events) {
  return sweep_groups(p, n, n_events) && n > kGroupWide &&
         (p.kernel_kind == CLUE_KERNEL_FLAT || n * ((n + 4095) / 4096) > 46000);
}

cudaError_t launch_density_group(int D, const RunParams& p, const SweepArgs& a, cudaStream_t st) {
  const bool wide = a.n <= kGroupWide;
  if (D == 2)
    return wide ? launch_kind<2, 32>(p, a, st) : launch_kind<2, 16>(p, a, st);
  return wide ? launch_kind<3, 32>(p, a, st) : launch_kind<3, 16>(p, a, st);
}

}  // namespace clue_impl
