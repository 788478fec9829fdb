"""Batches with one grid for all events have many more tiles than points; a warp of
the per-tile kernels (tile sort, cell layout) then takes several tiles at a time, a
lane each where they hold a few points. Compared with the checker bit for bit.
"""

import numpy as np
import pytest

import cluestering_b200 as clue
from cluestering_b200 import workloads as W
from tests.test_gpu_parity import check

pytestmark = pytest.mark.gpu


# tiles of the batch: 83,000 (2 a warp), 1.6 million (32 a warp)
@pytest.mark.parametrize("events,lo,hi", [(96, 200, 2000), (400, 200, 2400)])
@pytest.mark.parametrize("kernel,params,tags", [("flat", (0.5,), False), ("flat", (0.5,), True),
                                                ("gaussian", (0.8, 2.0), False)])
def test_shared_grid_of_many_events(events, lo, hi, kernel, params, tags):
    ev, sizes = W.batch_2d(events, lo, hi, seed=2000 + events)
    rng = np.random.default_rng(2001)
    w = rng.exponential(1.0, ev.n).astype(np.float32)
    check(ev.coords, w, 1.5, 5.0, 2.0, sizes=sizes, grid_mode=clue.GRID_SHARED, kernel=kernel, kernel_params=params,
          tags=rng.integers(0, 50, ev.n).astype(np.uint32) if tags else None, path="device")


@pytest.mark.parametrize("binning", [0, 1])
def test_shared_grid_of_many_events_3d(binning):
    rng = np.random.default_rng(2010)
    sizes = rng.integers(1, 2200, 120)
    evs = [W.layered_3d(max(60, int(s)), seed=2011 + k) for k, s in enumerate(sizes)]
    c = np.concatenate([e.coords for e in evs], axis=1)
    w = np.concatenate([e.weights for e in evs])
    algo = clue.Clusterer(3.0, 10.0, 4.0)
    algo.set_tuning(tile_binning=binning)
    check(c, w, 3.0, 10.0, 4.0, sizes=[e.n for e in evs], grid_mode=clue.GRID_SHARED, kernel="gaussian",
          kernel_params=(1.0, 1.0), clusterer=algo, path="device")


# Counting-sort binning puts every tile's ids in order: by a lane, by a warp or by a
# block's network of 2, 4, 8 or 16 ids a thread, beyond that by merging chunks.
@pytest.mark.parametrize("m", [2, 8, 9, 33, 129, 256, 257, 511, 512, 513, 1024, 1025, 2048, 2049, 4095, 4096, 4097, 9001])
def test_ids_of_a_tile_in_order(m):
    rng = np.random.default_rng(2100 + m)
    # the first event is one tile of m points in random index order, the second has
    # several, and the batch keeps the run off the one-cluster form
    c = rng.normal(0.0, 1.0, (2, m + 777)).astype(np.float32)
    w = rng.exponential(1.0, m + 777).astype(np.float32)
    algo = clue.Clusterer(0.3, 2.0, 0.5, points_per_tile=m)
    algo.set_tuning(tile_binning=0)
    from oracle import oracle as O
    from tests.test_gpu_parity import assert_identical, run_gpu
    g = run_gpu(c, w, 0.3, 2.0, 0.5, sizes=[m, 777], grid_mode=clue.GRID_PER_EVENT, clusterer=algo, path="device")
    assert_identical(g, O.make_clusters_batched(c, w, [m, 777], 0.3, 2.0, 0.5, shared_grid=False, points_per_tile=m,
                                                exp_mode=O.EXP_CLUE, n_threads=8))
