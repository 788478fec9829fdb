"""Coordinates and weights that are not ordinary numbers on the 2-D and 3-D Euclidean
path, in each of its forms (by the number of points: one cluster launch or the general
stages, 32 or 16 lanes per point or 32 points per warp), exponentials at the ends of their
ranges, and single events replayed from a CUDA graph. Compared with the checker."""

import numpy as np
import pytest

import cluestering_b200 as clue
from cluestering_b200 import workloads as W
from tests.test_gpu_parity import assert_identical, check, run_gpu, run_oracle

pytestmark = pytest.mark.gpu

SIZES = [900, 9000, 20000, 66000]


def event(D, n, seed):
    ev = W.blobs(n, max(1, n // 900), 0.0, 90.0, 1.0, 0.1, seed=seed, ndim=D, weights="exponential")
    order = np.random.default_rng(seed).permutation(n)
    return np.ascontiguousarray(ev.coords[:, order]), ev.weights[order]


def agree(a, b):
    """Two forms of one run agree; a NaN density may be any NaN."""
    assert np.array_equal(np.isnan(a["rho"]), np.isnan(b["rho"]))
    keep = ~np.isnan(a["rho"])
    assert np.array_equal(a["rho"][keep].view(np.int32), b["rho"][keep].view(np.int32))
    for k in ("nh", "seed", "ci"):
        assert np.array_equal(a[k], b[k])


def both_forms(c, w, *args, **kw):
    """The event on its own, and with 70 empty ones: the general stages, 32 points per
    warp and one lane per point."""
    one = run_gpu(c, w, *args, path="device", **kw)
    agree(one, run_gpu(c, w, *args, path="device", sizes=[c.shape[1]] + [0] * 70, grid_mode=clue.GRID_PER_EVENT, **kw))
    return one


@pytest.mark.parametrize("D", [2, 3])
@pytest.mark.parametrize("value,n", [(np.nan, n) for n in SIZES] + [(v, n) for v in (np.inf, -np.inf) for n in SIZES[:3]])
def test_coordinates(value, n, D):
    # (an infinite coordinate leaves the grid one tile)
    c, w = event(D, n, 11)
    c[0, [3, 40]] = value
    c[1, [40, 71]] = value
    check(c, w, 1.5, 3.0, 2.0, path="device")
    both_forms(c, w, 1.5, 3.0, 2.0)
    both_forms(c, w, 1.5, 3.0, 2.0, kernel="gaussian", kernel_params=(1.0, 1.0))


@pytest.mark.parametrize("kernel,params", [("flat", (0.5,)), ("exponential", (1.2, 0.7))])
@pytest.mark.parametrize("D", [2, 3])
@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("value", [-1.0, 0.0, -0.0, 1e-42, 3e38, np.inf, np.nan])
def test_weights(value, n, D, kernel, params):
    c, w = event(D, n, 12)
    w[::5] = value
    g = both_forms(c, w, 1.5, 3.0, 2.0, kernel=kernel, kernel_params=params)
    if np.isfinite(value):
        assert_identical(g, run_oracle(c, w, 1.5, 3.0, 2.0, kernel=kernel, kernel_params=params))


# Densities that are exponentials near the ends of their ranges: points without weight
# whose only neighbours lie at almost dc, with exponents around -79 and -100, the lines
# between the forms of the exponential, and a denominator that is a power of two or not.
@pytest.mark.parametrize("kernel,params,exponent", [("gaussian", (1.0, 1.0), lambda d: d * d / 2.0),
                                                    ("gaussian", (0.9, 1.3), lambda d: d * d / 1.62),
                                                    ("exponential", (1.2, 0.7), lambda d: 1.2 * d)])
@pytest.mark.parametrize("D,n", [(2, 901), (3, 9001), (2, 40001), (3, 70001)])
def test_exponents(D, n, kernel, params, exponent):
    rng = np.random.default_rng(n)
    for most in (40.0, 78.9, 79.1, 99.9, 100.1, 104.0):
        dc = 1.0
        while exponent(dc * 1.0001) < most:
            dc *= 1.0001
        c = rng.uniform(0.0, 0.004 * dc, (D, n))
        far = rng.random(n) < 0.02
        c[0, far] += 0.995 * dc
        c[1] += 3.0 * dc * (np.arange(n) // 1000)  # pairs of groups, far from one another
        w = np.where(far, rng.exponential(1.0, n) * 1e30, 0.0).astype(np.float32)
        g, o = check(c.astype(np.float32), w, dc, 1.0, dc, kernel=kernel, kernel_params=params, path="device")
        assert np.any(o.rho[~far] > 0.0) or most > 100.0


# A single event replayed from a graph: its tables are arguments of the captured kernels,
# and the last of them writes the seed count to the host. Few points, points enough for
# the density's second kernel, and one off the fast path.
@pytest.mark.parametrize("n,metric", [(1000, "euclidean"), (20000, "euclidean"), (9000, "manhattan")])
def test_graph_replay_of_a_single_event(n, metric):
    import torch
    dev, stream = torch.device("cuda", 0), torch.cuda.Stream()
    c, w = event(2, n, 13)
    pts = clue.PointsDevice(torch.from_numpy(c).to(dev), torch.from_numpy(w).to(dev))
    algo = clue.Clusterer(1.5, 3.0, 2.0)
    algo.set_graphs(True)
    measure = clue.EuclideanMetric() if metric == "euclidean" else clue.ManhattanMetric()
    crowded = c.copy()
    crowded[:, 5] = 1e5  # all others in one tile
    for k, (x, v) in enumerate([(c, w), (c, w), (c[:, ::-1] * 0.5, w), (crowded, w), (c, np.ones_like(w))]):
        pts.coords.copy_(torch.from_numpy(np.ascontiguousarray(x, np.float32)))
        pts.weights.copy_(torch.from_numpy(v))
        torch.cuda.synchronize()
        algo.make_clusters(pts, measure, clue.FlatKernel(0.5), stream=stream)
        assert algo.graph_replayed() == (k > 0)
        o = run_oracle(np.ascontiguousarray(x, np.float32), v, 1.5, 3.0, 2.0, metric=metric)
        assert algo.n_clusters() == o.n_clusters
        assert np.array_equal(algo.getSeeds(), o.seeds)
        stream.synchronize()
        assert_identical(dict(rho=pts.rho.cpu().numpy(), nh=pts.nearest_higher.cpu().numpy(),
                              seed=pts.is_seed.cpu().numpy(), ci=pts.cluster_index.cpu().numpy()), o)
