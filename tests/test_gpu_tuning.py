"""The autotuner leaves the launch choices that a run does not obey as they were: timing
them compares a run with itself, and what it happened to pick would stay in the workspace
for larger runs, which do obey it."""

import numpy as np
import pytest

import cluestering_b200 as clue
from cluestering_b200 import workloads as W

pytestmark = pytest.mark.gpu

DENSITY = ("density_union_x16_2d", "density_union_x16_3d", "density_shape")


@pytest.mark.parametrize("metric,D,n,m,grid,obeyed", [
    ("euclidean", 2, 3000, None, clue.GRID_PER_EVENT, ("cell_points",)),
    ("euclidean", 3, 65536, None, clue.GRID_PER_EVENT, ("cell_points",)),
    ("euclidean", 2, 20000, 1000, clue.GRID_PER_EVENT, ("cell_points", "tile_binning")),
    ("euclidean", 2, 20000, 1000, clue.GRID_SHARED, ("cell_points", "tile_binning", "label_jump_rounds")),
    ("euclidean", 2, 20000, 200, clue.GRID_PER_EVENT, ("cell_points", "tile_binning", "nh_shape") + DENSITY),
    ("euclidean", 3, 70000, None, clue.GRID_PER_EVENT, ("cell_points", "tile_binning", "label_jump_rounds") + DENSITY),
    ("manhattan", 2, 9000, None, clue.GRID_PER_EVENT, ()),
    ("manhattan", 2, 9000, 900, clue.GRID_PER_EVENT, ("tile_binning",)),
])
def test_autotuner_keeps_choices_the_run_does_not_obey(metric, D, n, m, grid, obeyed):
    import torch
    dev = torch.device("cuda", 0)
    ev = W.blobs(n, 20, 0.0, 80.0, 1.0, 0.1, seed=n + D, ndim=D, weights="exponential")
    pts = clue.PointsDevice(torch.from_numpy(ev.coords).to(dev), torch.from_numpy(ev.weights).to(dev))
    algo = clue.Clusterer(1.5, 5.0, 2.0)
    before = algo.get_tuning()
    sizes = None if m is None else np.full(n // m, m, np.uint32)
    chosen = algo.autotune(pts, clue.EuclideanMetric() if metric == "euclidean" else clue.ManhattanMetric(),
                           clue.FlatKernel(0.5), batch_item_sizes=sizes, grid_mode=grid, reps=1)
    assert algo.get_tuning() == chosen
    assert {k for k in chosen if chosen[k] != before[k]} <= set(obeyed)
