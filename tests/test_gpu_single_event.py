"""Single events at the edges of the one-cluster form (csrc/event.cu): its
stages before and after the sweeps each run as one thread-block cluster, for
events of at most 65,536 points and 2,560 tiles. Everything is compared with
the checker bit for bit, as in test_gpu_parity.py.
"""

import numpy as np
import pytest

import cluestering_b200 as clue
from cluestering_b200 import workloads as W
from tests.test_gpu_parity import check, run_gpu

pytestmark = pytest.mark.gpu


def shuffled(ev, seed):
    order = np.random.default_rng(seed).permutation(ev.n)
    return ev.coords[:, order], ev.weights[order]


# warps, rounds and blocks of the cluster that are empty, partly filled or full,
# and one point past the form's largest event
@pytest.mark.parametrize("n", [1, 2, 31, 33, 1024, 1025, 2048, 2049, 8193, 40007, 65535, 65536, 65537])
@pytest.mark.parametrize("weights", ["unit", "exponential"])
def test_event_sizes(n, weights):
    ev = W.blobs(n, max(1, n // 800), 0.0, 100.0, 1.0, 0.1, seed=900 + n % 89, weights=weights)
    c, w = shuffled(ev, n)
    check(c, w, 1.5, 5.0, 2.0, path="device")


@pytest.mark.parametrize("D,n", [(1, 30011), (3, 20011), (4, 9001), (5, 12007), (7, 5003), (10, 2049)])
def test_event_dimensions(D, n):
    ev = W.blobs(n, 9, 0.0, 40.0, 1.0, 0.1, seed=950 + D, weights="exponential", ndim=D)
    c, w = shuffled(ev, D)
    check(c, w, 0.2 if D == 1 else 1.5 if D < 4 else 2.5, 2.0, 2.0, path="device")


def test_event_with_every_option():
    ev = W.blobs(9001, 12, 0.0, 80.0, 1.0, 0.1, seed=960, weights="exponential")
    c, w = shuffled(ev, 1)
    rng = np.random.default_rng(961)
    check(c, w, 1.5, 5.0, 2.0, path="device", unc=rng.uniform(0.5, 1.5, ev.n).astype(np.float32),
          tags=rng.permutation(ev.n).astype(np.uint32),
          sigma=[rng.uniform(0.0, 1.0, ev.n).astype(np.float32), None])


def test_event_of_many_tiles_equals_the_batched_call():
    # more tiles than the one-cluster form holds (16 points a tile), and a batch
    # with an empty item, which never takes that form
    ev = W.blobs(45001, 60, 0.0, 100.0, 1.0, 0.1, seed=970, weights="exponential")
    c, w = shuffled(ev, 2)
    for ppt in (16, 24):  # 2,813 and 1,876 tiles asked for
        one = run_gpu(c, w, 1.5, 5.0, 2.0, path="device",
                      clusterer=clue.Clusterer(1.5, 5.0, 2.0, points_per_tile=ppt))
        two = run_gpu(c, w, 1.5, 5.0, 2.0, path="device", sizes=[ev.n, 0], grid_mode=clue.GRID_PER_EVENT,
                      clusterer=clue.Clusterer(1.5, 5.0, 2.0, points_per_tile=ppt))
        for k in ("rho", "nh", "seed", "ci"):
            assert np.array_equal(one[k].view(np.int32), two[k].view(np.int32)), (ppt, k)


def test_long_follower_chain():
    # 4,000 points on a line with rising weights: every point follows the next,
    # one chain through all of them
    n = 4000
    c = np.stack([np.arange(n, dtype=np.float32), np.zeros(n, np.float32)])
    g, _ = check(c, np.arange(1, n + 1, dtype=np.float32), 1.2, 1.0, 1.2, path="device")
    assert g["ci"].max() == 0
