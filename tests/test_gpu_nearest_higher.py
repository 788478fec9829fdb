"""The nearest-higher search with 32, 16, 8 and 1 lanes per point (chosen by the
dimension and the number of points), at sizes on both sides of every line, with
real-valued weights and on lattices of coincident points and few distinct tags,
where distances, densities and tags all tie and the first candidate in the
reference's visiting order wins. Compared with the checker bit for bit.
"""

import numpy as np
import pytest

from cluestering_b200 import workloads as W
from tests.test_gpu_parity import check

pytestmark = pytest.mark.gpu

SIZES = [(2, 4095), (2, 4097), (2, 16385), (2, 70001), (2, 262145), (3, 4096), (3, 16383), (3, 16387), (3, 70003)]


@pytest.mark.parametrize("D,n", SIZES)
def test_lattice_with_equal_tags(D, n):
    rng = np.random.default_rng(n)
    side = max(2, int(round((n / 2.0) ** (1.0 / D))))  # about two points per lattice site
    c = rng.integers(0, side, (D, n)).astype(np.float32)
    check(c, np.ones(n, np.float32), 1.0, 2.0, 1.5, path="device", tags=rng.integers(0, 3, n).astype(np.uint32))


@pytest.mark.parametrize("D,n", SIZES)
def test_blobs(D, n):
    ev = W.blobs(n, max(2, n // 800), 0.0, 100.0 if n < 1 << 18 else 400.0, 1.0, 0.1, seed=n, ndim=D,
                 weights="exponential")
    check(ev.coords, ev.weights, 1.5, 4.0, 2.0, 1.0, path="device")


@pytest.mark.parametrize("D,n", [(2, 3001), (2, 9001), (3, 3001), (3, 20011)])
def test_search_box_of_many_tiles(D, n):
    # a few points per tile and a radius of many tiles: more tiles in the box
    # than lanes, most of them empty
    rng = np.random.default_rng(n + D)
    import cluestering_b200 as clue
    from tests.test_gpu_parity import assert_identical, run_gpu
    from oracle import oracle as O
    c = rng.normal(0.0, 3.0, (D, n)).astype(np.float32)
    w = rng.exponential(1.0, n).astype(np.float32)
    g = run_gpu(c, w, 1.0, 2.0, 2.5, path="device", clusterer=clue.Clusterer(1.0, 2.0, 2.5, points_per_tile=4))
    assert_identical(g, O.make_clusters(c, w, 1.0, 2.0, 2.5, points_per_tile=4, exp_mode=O.EXP_CLUE, n_threads=8))


# One lane per point in 3-D, and the largest run with eight, every block shape: ties
# on a lattice, real weights, with and without tags.
@pytest.mark.parametrize("tags", [False, True])
@pytest.mark.parametrize("n,shape", [(524288, 0), (524289, 0), (600001, 1), (600001, 2)])
def test_large_runs_in_three_dimensions(n, shape, tags):
    import cluestering_b200 as clue
    rng = np.random.default_rng(n + shape)
    c = rng.uniform(0.0, 100.0, (3, n)).astype(np.float32)
    half = rng.random(n) < 0.5
    c[:, half] = np.round(c[:, half])
    w = np.where(half, 1.0, rng.exponential(1.0, n)).astype(np.float32)
    algo = clue.Clusterer(1.0, 2.0, 1.5)
    algo.set_tuning(nh_shape=shape)
    check(c, w, 1.0, 2.0, 1.5, path="device", clusterer=algo,
          tags=rng.integers(0, 3, n).astype(np.uint32) if tags else None)


# The lines above which even points have one lane per point and others eight: one event,
# and batches of events of at most 250 points, none of whose tiles can be large.
@pytest.mark.parametrize("D,n", [(2, 98304), (2, 98305), (3, 262144), (3, 262145)])
@pytest.mark.parametrize("crowd", [0, 400])
def test_even_points_of_one_event(D, n, crowd):
    rng = np.random.default_rng(n + crowd)
    c = rng.uniform(0.0, 200.0 if D == 2 else 60.0, (D, n))
    c[:, n - crowd:] = 10.0 + 0.05 * rng.normal(0.0, 1.0, (D, crowd))
    w = rng.exponential(1.0, n).astype(np.float32)
    check(c.astype(np.float32), w, 0.9, 2.0, 1.3, path="device")


@pytest.mark.parametrize("D,n,m", [(2, 16384, 16), (2, 32768, 250), (2, 32769, 250), (3, 32768, 100), (3, 32769, 100)])
def test_batches_of_small_events(D, n, m):
    import cluestering_b200 as clue
    rng = np.random.default_rng(n + m)
    c = rng.uniform(0.0, 20.0, (D, n))
    blob = rng.random(n) < 0.5
    c[:, blob] = 10.0 + 0.5 * rng.normal(0.0, 1.0, (D, int(blob.sum())))
    sizes = [m] * (n // m) + ([n % m] if n % m else [])
    w = rng.exponential(1.0, n).astype(np.float32)
    check(c.astype(np.float32), w, 0.9, 2.0, 1.3, path="device", sizes=sizes, grid_mode=clue.GRID_PER_EVENT,
          tags=rng.integers(0, 3, n).astype(np.uint32))
