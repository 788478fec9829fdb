"""The cluster -> points map on the device: one cluster launch for up to 65,536 points
and 2,560 clusters (csrc/event.cu), the general launches beyond, against the map of the
same labels built on the host. The labels are the caller's memory: ones that are no
cluster of the run are left out, as outliers are, whatever they hold."""

import numpy as np
import pytest

import cluestering_b200 as clue

pytestmark = pytest.mark.gpu


def sites(n, k, seed):
    """n points at k sites far apart: k clusters."""
    rng = np.random.default_rng(seed)
    s = np.concatenate([np.arange(k), rng.integers(0, k, n - k)])[rng.permutation(n)]
    side = int(np.ceil(np.sqrt(k)))
    c = np.stack([s // side, s % side]) * 10.0 + rng.uniform(0.0, 0.1, (2, n))
    return c.astype(np.float32)


def clustered(n, k, seed=5):
    import torch
    dev = torch.device("cuda", 0)
    pts = clue.PointsDevice(torch.from_numpy(sites(n, k, seed)).to(dev), torch.ones(n, device=dev))
    algo = clue.Clusterer(1.0, 0.5, 1.0)
    algo.make_clusters(pts)
    assert algo.n_clusters() == k
    return pts, algo


def check_map(pts, algo, k):
    lab = pts.cluster_index.cpu().numpy()
    offsets, members = (t.cpu().numpy() for t in algo.getClustersDevice())
    known = (lab >= 0) & (lab < k)
    order = np.argsort(np.where(known, lab, k), kind="stable")[: int(known.sum())]
    assert np.array_equal(offsets, np.concatenate([[0], np.cumsum(np.bincount(lab[known], minlength=k))]))
    assert np.array_equal(members, order)


@pytest.mark.parametrize("n,k", [(1, 1), (33, 2), (1024, 1023), (1025, 1024), (5000, 1025), (30000, 2559), (65535, 2560),
                                 (65536, 2561), (65536, 40), (65537, 40)])
def test_map(n, k):
    pts, algo = clustered(n, k)
    check_map(pts, algo, k)


# labels of another run of more clusters, of no run, and the type's ends
@pytest.mark.parametrize("n,k", [(700, 3), (20000, 40), (65536, 2600), (70001, 40)])
def test_labels_of_no_cluster_of_the_run_are_left_out(n, k):
    import torch
    pts, algo = clustered(n, k)
    lab = pts.cluster_index
    for at, value in enumerate([k, k + 1, n - 1, n, 2 ** 31 - 1, -2, -2 ** 31]):
        lab[at::11] = value
    check_map(pts, algo, k)
    lab.copy_(torch.arange(n, dtype=torch.int32, device=lab.device))  # every point its own label
    check_map(pts, algo, k)
