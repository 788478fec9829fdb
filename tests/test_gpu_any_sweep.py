"""The sweeps off the fast path (csrc/sweep_any.cu: a block per 32 points of one
tile, walking the union of their search boxes; csrc/sweep_any_point.cu: a warp per
point, up to 16,384 points) where the boxes are unusual, against the checker bit for
bit: items that span events, boxes that wrap round or cover the whole circle, boxes of
more tiles than are staged at a time, boxes that differ much in many dimensions, boxes
without the point's own tile, and weights or kernels whose out-of-range terms are not
zero. Each test runs below and above the line between the two forms.
"""

import math

import numpy as np
import pytest

import cluestering_b200 as clue
from cluestering_b200 import workloads as W
from oracle import oracle as O
from tests.test_gpu_parity import assert_identical, check, run_gpu, run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("events", [40, 200])
@pytest.mark.parametrize("mode", [clue.GRID_PER_EVENT, clue.GRID_SHARED])
def test_items_across_events(mode, events):
    ev, sizes = W.batch_2d(events, 1, 700, seed=31)
    w = np.random.default_rng(32).exponential(1.0, ev.n).astype(np.float32)
    check(ev.coords, w, 1.5, 3.0, 2.0, metric="manhattan", sizes=sizes, grid_mode=mode, path="device")


@pytest.mark.parametrize("n", [4099, 17001])
@pytest.mark.parametrize("r", [0.05, 0.7, 2.9, 7.0])
@pytest.mark.parametrize("wrapped", [[0, 1], [1, 0], [1, 1]])
def test_wrapped_boxes(r, wrapped, n):
    rng = np.random.default_rng(33)
    c = np.mod(np.stack([rng.normal(0.1, 0.8, n), rng.normal(6.2, 0.9, n)]), 2 * math.pi).astype(np.float32)
    w = rng.exponential(1.0, n).astype(np.float32)
    check(c, w, r, 2.0, 1.3 * r, metric="periodic_euclidean", metric_params=(2 * math.pi, 2 * math.pi),
          wrapped=wrapped, path="device")


@pytest.mark.parametrize("D,n,ppt,r", [(1, 3001, 2, 2.0), (2, 3001, 2, 12.0), (4, 6001, 4, 6.0), (5, 20011, 16, 2.0),
                                       (6, 5003, 4, 1.0), (1, 17001, 2, 0.5), (2, 17001, 2, 3.0), (4, 17001, 4, 4.0),
                                       (6, 17001, 4, 1.0), (2, 16384, 128, 1.0), (2, 16385, 128, 1.0)])
def test_boxes_of_many_tiles(D, n, ppt, r):
    rng = np.random.default_rng(34 + D)
    c = rng.uniform(0.0, 20.0, (D, n)).astype(np.float32)
    w = rng.exponential(1.0, n).astype(np.float32)
    g = run_gpu(c, w, r, 2.0, r, metric="chebyshev", path="device",
                clusterer=clue.Clusterer(r, 2.0, r, points_per_tile=ppt))
    assert_identical(g, O.make_clusters(c, w, r, 2.0, r, metric="chebyshev", points_per_tile=ppt,
                                        exp_mode=O.EXP_CLUE, n_threads=8))


@pytest.mark.parametrize("n", [3000, 17000])
def test_box_without_the_own_tile(n):
    # a radius beyond the int range of get_bin's conversion sends the box's upper
    # end to bin 0 (x86 conversion)
    ev = W.blobs(n, 6, 0.0, 30.0, 1.0, 0.1, seed=35, weights="exponential")
    check(ev.coords, ev.weights, 1.0, 3.0, 1e13, metric="manhattan", path="device")
    check(ev.coords, ev.weights, 3e12, 3.0, 1e13, metric="weighted_euclidean", metric_params=(1.0, 2.0), path="device")


@pytest.mark.parametrize("n", [2500, 17000])
@pytest.mark.parametrize("kernel,params", [("flat", (0.5,)), ("gaussian", (0.8, 2.0)), ("exponential", (1.2, 0.7))])
def test_infinite_and_nan_weights(kernel, params, n):
    # 0 * k * w of a candidate out of range is NaN for such a weight, and so is
    # every density whose search box holds it
    ev = W.blobs(n, 5, 0.0, 60.0, 1.0, 0.1, seed=36, weights="exponential")
    w = ev.weights.copy()
    w[[7, 900]] = np.inf
    w[1400] = np.nan
    kw = dict(metric="manhattan", kernel=kernel, kernel_params=params)
    g = run_gpu(ev.coords, w, 1.5, 3.0, 2.0, path="device", **kw)
    o = run_oracle(ev.coords, w, 1.5, 3.0, 2.0, **kw)
    assert np.isnan(o.rho).sum() > 100
    assert np.array_equal(np.isnan(g["rho"]), np.isnan(o.rho))
    keep = ~np.isnan(o.rho)
    assert np.array_equal(g["rho"][keep].view(np.int32), o.rho[keep].view(np.int32))
    assert np.array_equal(g["nh"], o.nearest_higher)
    assert np.array_equal(g["ci"], o.cluster_index)


@pytest.mark.parametrize("n", [6000, 17000])
def test_lattice_ties_and_equal_tags_in_four_dimensions(n):
    rng = np.random.default_rng(37)
    c = rng.integers(0, 7, (4, n)).astype(np.float32)
    check(c, np.ones(n, np.float32), 1.0, 2.0, 1.5, tags=rng.integers(0, 3, n).astype(np.uint32), path="device")


# The three forms and the lines between them: events of few points (a thread per point,
# in the sorted order up to 16,384 points), tiles of few points (one grid for a batch,
# many tiles per event), and runs beyond 65,536 points with and without tiles of more
# than 256, up to and past the form's largest run.
def _crowded(c, n, share, seed):
    """The last `share` of n points drawn together into one place."""
    k = int(n * share)
    c[:, n - k:] = 10.0 + 0.05 * np.random.default_rng(seed).normal(0.0, 1.0, (c.shape[0], k))
    return c.astype(np.float32)


@pytest.mark.parametrize("D,n,m,mode", [
    (2, 1600, 5, clue.GRID_PER_EVENT), (4, 16384, 16, clue.GRID_SHARED), (2, 16384, 64, clue.GRID_PER_EVENT),
    (3, 16385, 63, clue.GRID_PER_EVENT), (2, 32768, 127, clue.GRID_PER_EVENT), (2, 32768, 128, clue.GRID_PER_EVENT),
    (4, 40000, 200, clue.GRID_PER_EVENT), (2, 20000, 60, clue.GRID_SHARED), (1, 70000, 7000, clue.GRID_PER_EVENT),
    (3, 131072, 32768, clue.GRID_PER_EVENT)])
@pytest.mark.parametrize("crowd", [0.0, 0.02])  # none or the tile of the last events holds many points
def test_lines_between_the_forms(D, n, m, mode, crowd):
    rng = np.random.default_rng(n + m)
    c = rng.uniform(0.0, 20.0, (D, n)) * (1.0 if D > 1 else n / 2000.0)
    c = _crowded(c, n, crowd, n)
    w = rng.exponential(1.0, n).astype(np.float32)
    sizes = [m] * (n // m) + ([n % m] if n % m else [])
    if crowd and m < 1000:  # one larger event at the end
        k = -(-int(n * crowd) // m)
        sizes = sizes[:len(sizes) - k] + [sum(sizes[len(sizes) - k:])]
    check(c, w, 0.4, 2.0, 0.9, metric="manhattan", kernel="exponential", kernel_params=(1.2, 0.7), sizes=sizes,
          grid_mode=mode, tags=rng.integers(0, 50, n).astype(np.uint32), path="device")


@pytest.mark.parametrize("n", [65536, 65537, 1 << 20, (1 << 20) + 1])
@pytest.mark.parametrize("crowd", [0, 700])
def test_large_runs_off_the_fast_path(n, crowd):
    rng = np.random.default_rng(n)
    c = _crowded(rng.uniform(0.0, n / 100.0, (1, n)), n, crowd / n, 3)
    w = rng.exponential(1.0, n).astype(np.float32)
    check(c, w, 0.2, 2.0, 0.4, metric="manhattan", path="device")


# Stable binning of events that end inside the rounds loaded ahead, any number of
# dimensions (events of one point, of a round less or more one, of all rounds).
@pytest.mark.parametrize("D", [1, 2, 3, 4, 10])
def test_binning_of_tiny_events(D):
    sizes = [1, 31, 32, 33, 95, 96, 97, 127, 128, 129, 1023, 1024, 1025, 0, 5] * 3
    rng = np.random.default_rng(38 + D)
    c = rng.uniform(0.0, 4.0, (D, sum(sizes))).astype(np.float32)
    w = rng.exponential(1.0, c.shape[1]).astype(np.float32)
    check(c, w, 0.5, 2.0, 0.7, metric="chebyshev", sizes=sizes, grid_mode=clue.GRID_PER_EVENT, path="device")


# One event of even points at the sizes where the block of 8 warps gives way to the thread
# per point, and of sparse tiles in many dimensions, with and without a crowded tile.
@pytest.mark.parametrize("D,n,side", [(1, 81920, 4000.0), (3, 81921, 40.0), (4, 131072, 30.0), (4, 131073, 30.0),
                                      (6, 16385, 20.0), (6, 65537, 60.0), (7, 16385, 20.0)])
@pytest.mark.parametrize("crowd", [0, 400])
def test_single_event_lines(D, n, side, crowd):
    rng = np.random.default_rng(n + D)
    c = _crowded(rng.uniform(0.0, side, (D, n)), n, crowd / n, 5)
    w = rng.exponential(1.0, n).astype(np.float32)
    check(c, w, 0.5, 2.0, 0.9, metric="chebyshev", path="device")
