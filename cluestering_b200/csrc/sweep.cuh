// sweep.cuh — the local-density and nearest-higher sweeps.
#pragma once

#include "common.cuh"

namespace clue_impl {

// Some choices depend on whether a tile holds more than kLargeTilePoints points, which
// the host does not know: the kernels of both are launched, and one returns at once.
enum RunWhen { kNever, kAlways, kLargeTiles, kNoLargeTiles };

// Inputs and outputs of the two sweeps. Arrays prefixed with `s` are in
// tile-contiguous (sorted) order; plane d of sx/ssig starts at d * n.
struct SweepArgs {
  int64_t n;
  int64_t n_tiles;
  const EventDesc* events;
  const GridDesc* grids;
  const int32_t* tile_offset;
  const float* sx;
  const float* sw;
  const float* ssig;
  const float* sunc;
  const uint32_t* stag;
  const int32_t* perm;  // sorted position -> original index
  const int32_t* sevt;
  float* srho;
  // Processing order of each sweep: sorted positions grouped so that the
  // lanes of a warp share one search box (see launch_work_order).
  int32_t* work_dens;
  int32_t* work_nh;
  int32_t* cls_dens;  // scratch: box class per sorted position
  int32_t* cls_nh;
  // Work queues of the fast-path sweeps: [0] density, [1] nearest higher;
  // each counts the points or work items taken so far (k_gather, or the front of
  // a single event, resets both), so warps that finish early take the next.
  int32_t* queue;
  // Estimated times of the density, us, added up by the cell layout from its tiles: [0]
  // with lanes per point, [1] with 32 points per warp; density_streams compares them.
  // Null where lanes per point always do (density_by_load).
  float* load;
  // Tiles of more than 256 points (listed by the binning or the tile sort) and
  // their count: k_cells gives each of them a whole block. (The one-cluster form of a
  // single event only counts them, and only off the fast path: any_form.)
  const int32_t* large_tiles;
  const int32_t* large_count;
  // Exact-sum density (flat kernel): the density records again, in cell-layout
  // order, and per event four bounds on its contributions (smallest lowest-set-
  // bit exponent, largest neighbour contribution and largest weight as float
  // bits, and a flag for a negative or non-finite one) that decide whether the
  // event's sums are exact in any order. Null when the cell layout is off.
  float4* rec_cell;
  int32_t* event_exact;
  int32_t n_events;
  int32_t max_event_points;
  // Walk order of the cell layout (k_cells): walk[k] is the layout position
  // visited k-th, tile by tile, cells in strips of 4 rows so that consecutive
  // points are spatial neighbours. Orders the density work and the
  // nearest-higher threads. Null, like work_dens, when the sweeps take the points
  // in layout order (sweep_tile_blocks).
  int32_t* walk;
  bool tile_blocks;
  RunWhen nh_when;  // whether a launch of the nearest-higher search has the run
  // Packed candidate records of the fast path (D = 2 or 3).
  float4* rec_dens;  // {x, y, [z], v}: v = flat * w for the flat kernel, else w
  float4* rec_nh;    // D = 2: {x, y, rho, tag bits}; D = 3: {x, y, z, rho}
  uint32_t* rec_tag; // D = 3: tag of each record
  // outputs in original order
  float* out_rho;      // may be null
  int32_t* out_nh;     // required
  int32_t* out_seed;   // may be null
  int32_t* seed_flag;  // required
  // Nearest higher as a sorted position (the point itself when it has none):
  // the follower tree in the tile-contiguous layout, where chains stay local.
  int32_t* parent;
  // Cell layout of the nearest-higher search (null unless sweep_fast_path):
  // every tile is split into s^D cells (s per tile in cell_s, origin and
  // inverse cell width per dimension in cell_geom); the points of a tile are
  // reordered cell by cell inside the tile's range. A tile starting at sorted
  // position b keeps its cells in slots b .. b + s^D - 1 (s^D never exceeds
  // the tile's point count).
  // The cells are built for every fast-path run: the density sweep uses them to
  // skip out-of-reach candidates, and the nearest-higher search runs over them
  // (its records are in cell order).
  int32_t* nh_pos;        // sorted position -> layout position
  int32_t* nh_q;          // layout position -> sorted position
  int32_t* cell_slot;     // sorted position -> slot of its cell
  int32_t* cell_s;        // per tile
  float4* cell_geom;      // per tile: D = 2 {lo0, lo1, inv0, inv1}; D = 3 two entries
  CellInfo* cell_info;    // per slot
  float4* cell_box;       // per slot: bounding box of the members (D = 3: two entries)
  // Sweep statistics (null unless the run counts them): [0] density candidate
  // tests (a point testing one record), [1] density work items of 32 points, [2] nearest-
  // higher members tested, [3] cells checked, [4] cells whose members were tested.
  unsigned long long* stats;
  // Status word of the run: kernels with bounded waits set bits here.
  uint32_t* status;
};

// Whether a kernel launched for the case `when` has the run.
__device__ __forceinline__ bool runs_when(const SweepArgs& a, RunWhen when) {
  return when == kAlways || (*a.large_count > 0) == (when == kLargeTiles);
}

// True when the packed fast path applies: D = 2 or 3, Euclidean metric, no
// per-point sigma and no wrapped coordinate.
bool sweep_fast_path(const RunParams& p);

cudaError_t launch_work_order(int D, const RunParams& p, const SweepArgs& a, cudaStream_t st);
// The density with 16 or 32 lanes per point (density_group.cu), for fast-path runs of
// at most kGroupPoints points in at most 64 events, 32 above 49,152 points. Small events
// have few candidates to share among lanes: density, us, 32 points per warp / lanes, 65,536
// points in events of 16 12 / 48, of 256 23 / 49, of 512 29 / 49, of 1,024 40 / 50 (Gaussian
// 47 / 49 at 256, 113 / 54 at 1,024); 16,384 in events of 64 12 / 21, of 256 20 / 21, of 512
// 24 / 21; blobs, 22,742 points in 64 events 44 / 39, 33,129 in 40 74 / 68, 59,757 in 64 76 /
// 105 (ordered sums, one grid: 73 / 189).
constexpr int64_t kGroupPoints = 1 << 16, kGroupWide = 1 << 13;  // 32 lanes up to the latter
bool sweep_groups(const RunParams& p, int64_t n, int32_t n_events);
cudaError_t launch_density_group(int D, const RunParams& p, const SweepArgs& a, cudaStream_t st);
// Whether such a run may take 32 points per warp all the same (density_streams), and
// both kernels are launched.
bool density_by_load(const RunParams& p, int64_t n, int32_t n_events);
// In 3-D 32 points per warp take at least 3.4 ns a point, for the boxes of many tiles: a
// call of 65,536 points in 160 blobs 413 us with them and 292 with lanes, in 80 428 / 372,
// in 40 511 / 538, in 20 553 / 848 (loads 132 / 66, 229 / 143, 414 / 171, 775 / 405).
template <int D>
__device__ __forceinline__ bool density_streams(const SweepArgs& a) {
  return a.load && a.load[0] > fmaxf(a.load[1], D == 3 ? 3.4e-3f * (float)a.n : 0.0f) + 50.0f;
}
// Runs whose sweeps give every point a group of lanes (sweep_groups) take the
// points in layout order, and k_cells_tile lays the cells out with a block per tile;
// `walk` and `work_dens` are then null. Above kTileBlocks tiles (twice what the GPU holds
// at once) most hold too few points for a block of their own: gather, us, tile by warps /
// blocks, 16 events with one grid, 2,304 tiles: even points 17 / 22, blobs 28 / 17; 4,096
// tiles of 16 points 20 / 36. The one-cluster form of a single event, which leaves no
// coordinate planes, has no more than that.
constexpr int64_t kTileBlocks = 2560;
bool sweep_tile_blocks(const RunParams& p, int64_t n, int64_t n_tiles, int32_t n_events);
// Lanes per point of the nearest-higher search on the fast path: `lanes` where tiles hold
// more than kLargeTilePoints points or always (when), else one.
struct NearestForm {
  int lanes;
  RunWhen when;
};
NearestForm nearest_form(int D, int64_t n, int32_t n_events, int32_t max_event_points);
// The sweeps off the fast path: any number of dimensions, metric, kernel and
// option. Three forms, chosen by any_form (sweep_any.cu): a warp per point
// (sweep_any_point.cu), a block of 8 warps per 32 points (sweep_any.cu) and a thread
// per point (sweep_any_thread.cu).
struct AnyForm {
  RunWhen point = kNever, block = kNever, thread = kNever;
  bool work_order = false;  // k_work_order runs first
};
AnyForm any_form(int D, const SweepArgs& a);
cudaError_t launch_density_any(int D, const RunParams& p, const SweepArgs& a, cudaStream_t st);
cudaError_t launch_nearest_higher_any(int D, const RunParams& p, const SweepArgs& a, cudaStream_t st);
cudaError_t launch_sweep_point(bool density, int D, const RunParams& p, const SweepArgs& a, cudaStream_t st);
cudaError_t launch_sweep_thread(bool density, int D, const RunParams& p, const SweepArgs& a, RunWhen when,
                                cudaStream_t st);
cudaError_t launch_density(int D, const RunParams& p, const SweepArgs& a, cudaStream_t st);
cudaError_t launch_nearest_higher(int D, const RunParams& p, const SweepArgs& a, cudaStream_t st);

}  // namespace clue_impl
