"""The density sweep's forms (16 or 32 lanes per point, 32 points per warp) where
the lists of candidates are unusual, against the checker bit for bit: tiles of more
points than a candidate bitmap covers, search boxes of many tiles, events with exact
and with ordered sums in one run, coordinates far from the origin, degenerate tiles.
"""

import numpy as np
import pytest

import cluestering_b200 as clue
from cluestering_b200 import workloads as W
from oracle import oracle as O
from tests.test_gpu_parity import assert_identical, check, run_gpu

pytestmark = pytest.mark.gpu

KERNELS = [("flat", (0.5,), "unit"), ("flat", (0.3,), "exponential"), ("gaussian", (0.7, 1.5), "exponential"),
           ("exponential", (1.1, 0.9), "unit")]
# both sides of the lines between the forms
SIZES = [700, 8192, 8193, 65536, 65537]


def event(D, n, weights, seed):
    ev = W.blobs(n, max(1, n // 3000), 0.0, 60.0, 1.0, 0.15, seed=seed, ndim=D, weights=weights)
    order = np.random.default_rng(seed).permutation(n)
    return np.ascontiguousarray(ev.coords[:, order]), ev.weights[order]


def check_ppt(c, w, dc, rhoc, dm, ppt, **kw):
    g = run_gpu(c, w, dc, rhoc, dm, path="device", clusterer=clue.Clusterer(dc, rhoc, dm, points_per_tile=ppt), **kw)
    assert_identical(g, O.make_clusters(c, w, dc, rhoc, dm, points_per_tile=ppt, exp_mode=O.EXP_CLUE, n_threads=8,
                                        **kw))


@pytest.mark.parametrize("kernel,params,weights", KERNELS)
@pytest.mark.parametrize("D", [2, 3])
@pytest.mark.parametrize("n", SIZES)
def test_shuffled_blobs(D, n, kernel, params, weights):
    c, w = event(D, n, weights, 1000 + n % 97 + D)
    check(c, w, 1.2, 3.0, 1.5, kernel=kernel, kernel_params=params, path="device")


@pytest.mark.parametrize("kernel,params,weights", KERNELS)
@pytest.mark.parametrize("D,n,ppt", [(2, 9000, 20000), (3, 9000, 20000), (2, 70000, 30000), (3, 70000, 12000)])
def test_tiles_larger_than_the_bitmap(D, n, ppt, kernel, params, weights):
    c, w = event(D, n, weights, 1100 + D)
    check_ppt(c, w, 0.4, 3.0, 0.5, ppt, kernel=kernel, kernel_params=params)


@pytest.mark.parametrize("kernel,params,weights", KERNELS)
@pytest.mark.parametrize("D,n,r", [(2, 3000, 6.0), (3, 3000, 9.0), (2, 66000, 1.5), (3, 66000, 4.0)])
def test_search_boxes_of_many_tiles(D, n, r, kernel, params, weights):
    c, w = event(D, n, weights, 1200 + D)
    check_ppt(c, w, r, 3.0, r, 4, kernel=kernel, kernel_params=params)


@pytest.mark.parametrize("scale", [1, 12])
@pytest.mark.parametrize("mode", [clue.GRID_PER_EVENT, clue.GRID_SHARED])
def test_exact_and_ordered_events_together(scale, mode):
    ev, sizes = W.batch_2d(24, 60, 1500 * scale, seed=1300)
    w = ev.weights.copy()
    begin = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    rng = np.random.default_rng(1301)
    for e in range(0, len(sizes), 2):  # every other event
        w[begin[e]:begin[e + 1]] = rng.exponential(1.0, int(sizes[e])).astype(np.float32)
    check(ev.coords, w, 1.5, 3.0, 2.0, sizes=sizes, grid_mode=mode, path="device")


@pytest.mark.parametrize("kernel,params,weights", KERNELS)
@pytest.mark.parametrize("n", [5000, 66000])
def test_far_from_the_origin(n, kernel, params, weights):
    # the tiles' edges round to 1/16 here, a quarter of the radius
    c, w = event(2, n, weights, 1400)
    c = c + np.array([[9e5], [-7e5]], np.float32)
    check(c, w, 0.25, 3.0, 0.5, kernel=kernel, kernel_params=params, path="device")


@pytest.mark.parametrize("kernel,params,weights", KERNELS)
def test_points_on_a_line_and_coincident_points(kernel, params, weights):
    rng = np.random.default_rng(1500)
    n = 6000
    w = np.ones(n, np.float32) if weights == "unit" else rng.exponential(1.0, n).astype(np.float32)
    c = np.stack([np.full(n, 3.5), rng.normal(0.0, 4.0, n)]).astype(np.float32)  # tiles of no width
    check(c, w, 0.3, 3.0, 0.5, kernel=kernel, kernel_params=params, path="device")
    c = np.repeat(rng.uniform(0.0, 5.0, (2, 12)), n // 12, axis=1).astype(np.float32)
    check(c, w, 0.3, 3.0, 0.5, kernel=kernel, kernel_params=params, path="device")


# One block lays out a tile: few cells (boxes grown by atomics), more cells than it keeps
# boxes for, more points than it keeps; coordinates of both signs, zeros of both signs
# and all points of a cell at one place.
@pytest.mark.parametrize("cell_points", [1, 2, 8])
@pytest.mark.parametrize("n", [3, 1023, 1100, 2047, 2049, 5000])
@pytest.mark.parametrize("D", [2, 3])
def test_cell_boxes_of_one_tile(D, n, cell_points):
    rng = np.random.default_rng(n + D)
    c = rng.uniform(-4.0, 4.0, (D, n)).astype(np.float32)
    c[:, rng.random(n) < 0.2] = np.float32(-1.25)
    c[0, ::7] = np.float32(0.0)
    c[1, ::11] = np.float32(-0.0)
    w = rng.exponential(1.0, n).astype(np.float32)
    clusterer = clue.Clusterer(0.3, 2.0, 0.9, points_per_tile=2 * n)
    clusterer.set_tuning(cell_points=cell_points)
    g = run_gpu(c, w, 0.3, 2.0, 0.9, path="device", clusterer=clusterer)
    assert_identical(g, O.make_clusters(c, w, 0.3, 2.0, 0.9, points_per_tile=2 * n, exp_mode=O.EXP_CLUE, n_threads=8))


# Crowded tiles, where the density takes 32 points per warp below 65,537 points too: an
# outlier that leaves all other points one tile or one cell, and a radius over the whole
# extent; sizes on both sides of the lines (8,192 points; 12,288 with the smooth kernels),
# and a batch of as many tiles as k_cells lays out.
@pytest.mark.parametrize("kernel,params,weights", KERNELS + [("gaussian", (1.0, 1.0), "exponential")])
@pytest.mark.parametrize("D,n,outlier,r", [(2, 8192, 3e3, 1.2), (2, 8193, 3e5, 1.2), (2, 12288, 3e5, 1.2),
                                           (3, 12289, 3e4, 1.5), (2, 20011, 3e3, 1.2), (3, 20011, 3e5, 1.5),
                                           (2, 20011, None, 90.0), (3, 9001, None, 25.0)])
def test_crowded_tiles(D, n, outlier, r, kernel, params, weights):
    c, w = event(D, n, weights, 1600 + D)
    if outlier:
        c[:, n // 2] = outlier
    check(c, w, r, 3.0, r if r < 20.0 else 1.0, kernel=kernel, kernel_params=params, path="device")


@pytest.mark.parametrize("weights", ["unit", "exponential"])
def test_largest_crowded_tile(weights):
    c, w = event(2, 65536, weights, 1650)
    c[:, 7] = 3e5
    check(c, w, 1.2, 3.0, 1.2, path="device")


@pytest.mark.parametrize("kernel,params,weights", KERNELS)
@pytest.mark.parametrize("mode", [clue.GRID_PER_EVENT, clue.GRID_SHARED])
def test_crowded_tiles_in_a_batch(mode, kernel, params, weights):
    sizes = [4000, 9000, 300, 12000, 1, 2500]
    c, w = event(2, sum(sizes), weights, 1700)
    c[:, 10], c[:, 5000] = 2e4, -2e4
    g = run_gpu(c, w, 1.2, 3.0, 1.5, kernel=kernel, kernel_params=params, sizes=sizes, grid_mode=mode, path="device",
                clusterer=clue.Clusterer(1.2, 3.0, 1.5, points_per_tile=96))
    assert_identical(g, O.make_clusters_batched(c, w, sizes, 1.2, 3.0, 1.5, shared_grid=mode == clue.GRID_SHARED,
                                                points_per_tile=96, kernel=kernel, kernel_params=params,
                                                exp_mode=O.EXP_CLUE, n_threads=8))


# Small events: lanes per point up to 64 events (density 32 above 49,152 points; nearest
# higher 64 in 2-D, 128 in 3-D, half of that above 65,536 points), beyond that one lane per
# point unless a tile holds more than 256 points.
@pytest.mark.parametrize("kernel,params,weights", KERNELS[1:3])
@pytest.mark.parametrize("D,events,m", [(2, 63, 90), (2, 64, 90), (2, 65, 90), (3, 65, 40), (3, 128, 40), (3, 129, 40),
                                        (2, 32, 2049), (2, 33, 2049), (3, 64, 1025), (3, 65, 1025),
                                        (2, 32, 1700), (2, 33, 1700)])
@pytest.mark.parametrize("crowd", [False, True])
def test_batches_of_small_events(D, events, m, crowd, kernel, params, weights):
    rng = np.random.default_rng(1800 + events)
    sizes = rng.integers(1, 2 * m, events)
    sizes[-1] += max(0, m * events - sizes.sum())
    sizes[0] = 900
    c = rng.uniform(0.0, 6.0, (D, int(sizes.sum()))).astype(np.float32)
    if crowd:  # one tile of the first event
        c[:, 300:900] = 3.0 + 0.01 * c[:, 300:900]
    w = rng.exponential(1.0, c.shape[1]).astype(np.float32)
    tags = rng.integers(0, 9, c.shape[1]).astype(np.uint32) if kernel == "flat" else None
    check(c, w, 0.8, 2.0, 1.1, kernel=kernel, kernel_params=params, sizes=sizes, tags=tags,
          grid_mode=clue.GRID_PER_EVENT, path="device")
