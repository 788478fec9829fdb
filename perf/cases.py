"""Performance cases: the clustering calls that programs make of this package.

listed() and draw() describe cases as dicts of plain values, prepare() makes a
case's inputs and handle on the GPU (on the host for the calls that take host
points), run() makes one pass through the public entry points, work() states
what a pass cannot do without and exact() what it returns in 64-bit arithmetic.

The events are those of the package's workloads, made on the GPU: isotropic
Gaussian blobs plus uniform noise, and layered showers in a 3-D detector.
Every case has its own Clusterer with the default settings, which the program
keeps from call to call.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import cluestering_b200 as clue
from cluestering_b200 import api

LAYERS, SHOWERS, DEPTH_RATIO = 50, 30, 0.9
NOISE_2D, NOISE_3D = 0.1, 0.15
EXACT_POINTS = 1 << 21  # exact() takes seconds up to here


# -- the cases ------------------------------------------------------------------


def _event(n, **kw):
    """One event: 20 blobs of width 1 for each 16,384 points in [0, 100]^2, unit
    weights, flat kernel, as device arrays."""
    c = dict(call="cluster", where="device", shape="blobs", ndim=2, n=n, events=1, lo=n, hi=n,
             grid="per_event", blobs_per_16k=20, extent=100.0, sigma=1.0, weights="unit",
             shuffled=False, dc=1.5, rhoc=5.0, dm=1.5, kernel="flat", periodic=False, options=False)
    c.update(kw)
    return c


def _field(n, **kw):
    """A large field: a fixed density of blobs (2,000 in [0, 1000]^2 for 1,048,576
    points) with exponential weights."""
    return _event(n, blobs_per_16k=31.25, extent=1000.0 * math.sqrt(n / 1048576.0),
                  weights="exponential", rhoc=8.0, dm=2.0, **kw)


def _layered(n, **kw):
    """Hits of showers in a detector of 50 layers, Gaussian kernel, energies as weights."""
    return _event(n, shape="layered", ndim=3, dc=3.0, rhoc=10.0, dm=4.0, kernel="gaussian",
                  weights="lognormal", **kw)


def _batch(events, lo, hi, **kw):
    """Events of sizes log-uniform in [lo, hi] clustered by one call."""
    return _event(0, events=events, lo=lo, hi=hi, **kw)


def _score(n, **kw):
    """Centroids and silhouettes of a clustering that is at hand."""
    return _event(n, call="score", rhoc=15.0, **kw)


def _towers(n, **kw):
    """Pseudorapidity and azimuth: 20 jets, the azimuth periodic."""
    return _event(n, blobs_per_16k=20 * 16384.0 / n, extent=2.0 * math.pi, sigma=0.1, dc=0.1, rhoc=5.0,
                  dm=0.15, periodic=True, weights="exponential", shuffled=True, **kw)


def listed():
    return [
        # the smallest call: one event of a trigger or of a test beam, latency alone
        _event(1024, name="event_1k"),
        # an ordinary single event, the reference benchmark's middle size
        _event(16384, name="event_16k"),
        # a large field of measurements with real-valued weights
        _field(1048576, name="field_1m"),
        # calorimeter hits of one event as a reconstruction program holds them: host arrays
        _layered(10000, where="pageable", name="layered_10k_host"),
        # a high-occupancy calorimeter event on the device
        _layered(262144, name="layered_262k"),
        # the headline batch: many events of mixed sizes, resident on the device
        _batch(4096, 256, 65536, name="batch_4096"),
        # the same kind of batch delivered by a data loader in pinned memory
        _batch(1024, 256, 65536, where="pinned", name="batch_1024_host"),
        # small events of odd sizes in the reference's batched form (one grid for the batch)
        _batch(301, 300, 5001, grid="shared", weights="exponential", shuffled=True, name="batch_301_shared"),
        # jets in pseudorapidity and azimuth: periodic metric and wrapped coordinate
        _towers(32768, name="towers_32k"),
        # per-point density uncertainties and tags, exponential kernel, an odd size
        _event(50021, weights="exponential", kernel="exponential", options=True, shuffled=True,
               rhoc=8.0, dm=2.0, name="tagged_50k"),
        # feature vectors of four dimensions
        _event(16384, ndim=4, dc=3.0, dm=3.0, weights="exponential", name="features_4d"),
        # scoring a clustering: the cluster map, centroids and silhouettes
        _score(32768, name="score_32k"),
    ]


def draw(rng):
    def size(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))

    family = rng.randrange(10)
    shuffled = rng.random() < 0.5
    where = rng.choice(["device", "device", "pageable"])
    if family == 0:
        return _event(size(256, 262144), where=where, shuffled=shuffled)
    if family == 1:
        return _event(size(256, 262144), where=where, shuffled=shuffled, weights="exponential",
                      kernel=rng.choice(["flat", "gaussian", "exponential"]), dm=rng.choice([1.5, 2.0, 3.0]))
    if family == 2:
        return _field(size(65536, 2097152), shuffled=shuffled)
    if family == 3:
        return _layered(size(1024, 262144), where=where, shuffled=shuffled)
    if family == 4:
        return _batch(size(16, 2048), 256, size(2048, 65536), shuffled=shuffled,
                      weights=rng.choice(["unit", "unit", "exponential"]))
    if family == 5:
        return _batch(size(16, 1024), 256, size(2048, 65536), where="pinned", shuffled=shuffled)
    if family == 6:
        return _batch(size(8, 512), 256, size(512, 8192), grid="shared", shuffled=shuffled,
                      weights=rng.choice(["unit", "exponential"]))
    if family == 7:
        return _towers(size(1024, 131072))
    if family == 8:
        return _event(size(1024, 131072), weights="exponential", options=True, shuffled=shuffled, dm=2.0,
                      kernel=rng.choice(["flat", "exponential"]))
    if rng.random() < 0.5:
        return _event(size(1024, 32768), ndim=rng.choice([1, 4, 5]), dc=3.0, dm=3.0, weights="exponential",
                      shuffled=shuffled)
    return _score(size(2048, 65536), shuffled=shuffled)


# -- inputs -----------------------------------------------------------------------


def _kernel(case):
    return {"flat": clue.FlatKernel(0.5), "gaussian": clue.GaussianKernel(1.0, 1.0),
            "exponential": clue.ExponentialKernel(1.2, 0.7)}[case["kernel"]]


def _sizes(case):
    """Points of each event: a batch's sizes belong to the case."""
    if case["events"] == 1:
        return np.array([case["n"]], np.int64)
    rng = np.random.default_rng([case["events"], case["lo"], case["hi"]])
    u = rng.uniform(math.log(case["lo"]), math.log(case["hi"] + 1), case["events"])
    return np.minimum(np.floor(np.exp(u)), case["hi"]).astype(np.int64)


def _blob_count(case, n):
    return np.maximum(1, np.round(case["blobs_per_16k"] * np.asarray(n) / 16384.0)).astype(np.int64)


def _points(case, seed):
    """(coords (D, n), weights (n,)) on the GPU and the event sizes."""
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    sizes = _sizes(case)
    n, D = int(sizes.sum()), case["ndim"]

    def uniform(*shape):
        return torch.rand(*shape, generator=g, device=dev)

    def normal(*shape):
        return torch.randn(*shape, generator=g, device=dev)

    event = torch.repeat_interleave(torch.arange(len(sizes), device=dev), torch.as_tensor(sizes, device=dev))
    if case["shape"] == "layered":
        n_noise = int(round(n * NOISE_3D))
        share = DEPTH_RATIO ** np.arange(LAYERS)
        per_layer = np.floor((n - n_noise) * share / share.sum()).astype(np.int64)
        per_layer[0] += n - n_noise - per_layer.sum()
        z = torch.repeat_interleave(torch.arange(LAYERS, device=dev), torch.as_tensor(per_layer, device=dev))
        centre = uniform(SHOWERS, 2) * 200.0 - 100.0
        which = torch.randint(0, SHOWERS, (n - n_noise,), generator=g, device=dev)
        xy = centre[which] + 2.0 * normal(n - n_noise, 2)
        z = torch.cat([z, torch.randint(0, LAYERS, (n_noise,), generator=g, device=dev)]).float()
        xy = torch.cat([xy, uniform(n_noise, 2) * 200.0 - 100.0])
        coords = torch.stack([xy[:, 0], xy[:, 1], z])
        weights = torch.exp(normal(n)) * DEPTH_RATIO ** z
        weights[n - n_noise:] = 0.1
    else:
        blobs = _blob_count(case, sizes)
        per_blob = np.floor(sizes * (1.0 - NOISE_2D) / blobs).astype(np.int64)
        begin = np.concatenate([[0], np.cumsum(sizes)[:-1]])
        first = np.concatenate([[0], np.cumsum(blobs)[:-1]])
        to = lambda a: torch.as_tensor(a, device=dev)  # noqa: E731
        blob = (torch.arange(n, device=dev) - to(begin)[event]) // torch.clamp(to(per_blob)[event], min=1)
        in_blob = blob < to(blobs)[event]
        count = int(blobs.sum())
        centre = uniform(D, count)
        if case["call"] == "score":  # well separated blobs: centres around the points of a lattice
            side = math.ceil(math.sqrt(count))
            k = torch.arange(count, device=dev)
            centre = (torch.stack([k // side, k % side]) + 0.4 + 0.2 * centre) / side
        centre = centre * case["extent"]
        at = torch.where(in_blob, to(first)[event] + blob, 0)
        coords = torch.empty((D, n), device=dev)
        for d in range(D):
            coords[d] = torch.where(in_blob, centre[d][at] + case["sigma"] * normal(n), uniform(n) * case["extent"])
        if case["periodic"]:  # the last coordinate is an angle in [0, 2 pi)
            coords[D - 1] = torch.remainder(coords[D - 1], 2.0 * math.pi)
        weights = -torch.log1p(-uniform(n)) if case["weights"] == "exponential" else torch.ones(n, device=dev)
    if case["shuffled"]:  # in no order inside each event
        order = torch.argsort(event.double() + uniform(n).double())
        coords, weights = coords[:, order], weights[order]
    return coords.float().contiguous(), weights.float().contiguous(), sizes


def _host_array(t, pinned):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=pinned)
    h.copy_(t)
    return h.numpy()


def prepare(case, seed):
    coords, weights, sizes = _points(case, seed)
    n = coords.shape[1]
    algo = clue.Clusterer(case["dc"], case["rhoc"], case["dm"])
    state = {"case": case, "algo": algo, "kernel": _kernel(case), "metric": None, "sizes": None}
    if case["periodic"]:
        algo.setWrappedCoordinates([0] * (case["ndim"] - 1) + [1])
        state["metric"] = clue.PeriodicEuclideanMetric([0.0] * (case["ndim"] - 1) + [2.0 * math.pi])
    if case["events"] > 1:
        state["sizes"] = sizes.astype(np.uint32)
    if case["where"] == "device":
        extra = {}
        if case["options"]:
            g = torch.Generator(device=coords.device)
            g.manual_seed(seed + 1)
            extra["density_uncertainty"] = 1.0 + 0.3 * torch.rand(n, generator=g, device=coords.device)
            extra["tags"] = torch.randperm(n, generator=g, device=coords.device).int()
        state["points"] = clue.PointsDevice(coords, weights, **extra)
    else:
        pinned = case["where"] == "pinned"
        labels = torch.full((n,), -1, dtype=torch.int32)
        state["points"] = clue.PointsHost(_host_array(coords, pinned), _host_array(weights, pinned),
                                          cluster_index=_host_array(labels, pinned))
    if case["call"] == "score":
        algo.make_clusters(state["points"], kernel=state["kernel"])
    return state


# -- one pass -----------------------------------------------------------------------


def run(state):
    case, algo, points = state["case"], state["algo"], state["points"]
    if case["call"] == "score":
        return {"centroids": api.cluster_centroids(points, algo),
                "weighted": api.weighted_cluster_centroids(points, algo),
                "silhouette": api.silhouette_scores(points, algo)}
    grid = clue.GRID_SHARED if case["grid"] == "shared" else clue.GRID_PER_EVENT
    algo.make_clusters(points, state["metric"], state["kernel"], batch_item_sizes=state["sizes"], grid_mode=grid)
    if case["where"] != "device":
        return {"cluster_index": points.cluster_index}
    return {"rho": points.rho, "nearest_higher": points.nearest_higher, "is_seed": points.is_seed,
            "cluster_index": points.cluster_index}


def _pairs(case):
    """Pairs of points of one event within dc, both orders, from the distributions."""
    sizes = _sizes(case).astype(np.float64)
    if case["shape"] == "layered":
        n = sizes.sum()
        share = DEPTH_RATIO ** np.arange(LAYERS)
        share *= n * (1.0 - NOISE_3D) / (share.sum() * SHOWERS)  # hits of a shower in each layer
        dc2, total = case["dc"] ** 2, 0.0
        for dz in range(-int(case["dc"]), int(case["dc"]) + 1):
            near = 1.0 - math.exp(-(dc2 - dz * dz) / 16.0)
            total += near * float(sum(share[z] * share[z + dz] for z in range(LAYERS) if 0 <= z + dz < LAYERS))
        return float(SHOWERS * total + n)
    m = sizes * (1.0 - NOISE_2D) / _blob_count(case, sizes)
    u, D = (case["dc"] / case["sigma"]) ** 2 / 4.0, case["ndim"]
    near = {1: math.erf(math.sqrt(u)), 2: 1.0 - math.exp(-u), 4: 1.0 - math.exp(-u) * (1.0 + u),
            5: math.erf(math.sqrt(u)) - math.exp(-u) * (2.0 + 4.0 * u / 3.0) * math.sqrt(u / math.pi)}[D]
    ball = {1: 2.0, 2: math.pi, 4: math.pi ** 2 / 2.0, 5: 8.0 * math.pi ** 2 / 15.0}[D] * case["dc"] ** D
    return float((sizes * (m * near + sizes * NOISE_2D * ball / case["extent"] ** D)).sum())


def work(case):
    n, D = float(_sizes(case).sum()), case["ndim"]
    if case["call"] == "score":
        # every point against every clustered point: a distance, its root and a sum
        return {"bytes": 4.0 * n * (D + 3), "flops": (1.0 - NOISE_2D) * n * n * (3 * D + 1)}
    outputs = 4 if case["where"] == "device" else 1
    inputs = D + 1 + (2 if case["options"] else 0)
    # each pair in range adds to a density: its distance and its contribution
    return {"bytes": 4.0 * n * (inputs + outputs), "flops": _pairs(case) * (3 * D + 1)}


# -- the same in 64 bits ------------------------------------------------------------


def _blocks(case, coords, sizes, rows=2048):
    """(i0, i1, j0, j1, d2) over the points in the order of the first coordinate
    (events one after another): every pair of an event within max(dc, dm) is in some block."""
    x = coords.double()
    reach = max(case["dc"], case["dm"]) * 1.001
    span = float(x[0].max() - x[0].min()) + 2.0 * reach
    event = torch.repeat_interleave(torch.arange(len(sizes), device=x.device), torch.as_tensor(sizes, device=x.device))
    line = x[0] - x[0].min() + event * span
    order = torch.argsort(line)
    line, x = line[order], x[:, order]
    starts = torch.arange(0, line.numel(), rows, device=x.device)
    ends = torch.clamp(starts + rows, max=line.numel())
    lo = torch.searchsorted(line, line[starts] - reach).tolist()
    hi = torch.searchsorted(line, line[ends - 1] + reach, right=True).tolist()
    event = event[order]

    def blocks():
        for i0, i1, j0, j1 in zip(starts.tolist(), ends.tolist(), lo, hi):
            d2 = torch.zeros((i1 - i0, j1 - j0), dtype=torch.float64, device=x.device)
            for d in range(case["ndim"]):
                diff = x[d, i0:i1, None] - x[d, None, j0:j1]
                if case["periodic"] and d == case["ndim"] - 1:
                    diff = diff.abs()
                    diff = torch.minimum(diff, 2.0 * math.pi - diff)
                d2 += diff * diff
            if len(sizes) > 1:
                d2[event[i0:i1, None] != event[None, j0:j1]] = math.inf
            yield i0, i1, j0, j1, d2

    return order, blocks


def _density(case, coords, weights, sizes):
    order, blocks = _blocks(case, coords, sizes)
    w = weights.double()[order]
    # the radius is a 32-bit number in the path: points at that distance are in range
    dc = float(np.float32(case["dc"]))
    rho = torch.empty_like(w)
    for i0, i1, j0, j1, d2 in blocks():
        if case["kernel"] == "flat":
            k = torch.full_like(d2, 0.5)
        elif case["kernel"] == "gaussian":
            k = torch.exp(-d2 / 2.0)
        else:
            k = 0.7 * torch.exp(-1.2 * torch.sqrt(d2))
        k[d2 > dc * dc] = 0.0
        i = torch.arange(i0, i1, device=k.device)
        k[i - i0, i - j0] = 1.0
        rho[i0:i1] = k @ w[j0:j1]
    out = torch.empty_like(rho)
    out[order] = rho
    return out


def _labels(case, coords, weights, sizes):
    """Cluster of each point, -1 for outliers, from the definition of the algorithm."""
    rho = _density(case, coords, weights, sizes)
    order, blocks = _blocks(case, coords, sizes)
    r = rho[order]
    seed_like = r >= case["rhoc"]
    best = torch.full_like(order, -1)
    eff = torch.where(seed_like, case["dc"], case["dm"])
    for i0, i1, j0, j1, d2 in blocks():
        ri, rj = r[i0:i1, None], r[None, j0:j1]
        higher = (rj > ri) | ((rj == ri) & (order[None, j0:j1] > order[i0:i1, None]))
        d2 = torch.where(higher & (d2 <= (eff[i0:i1, None]) ** 2), d2, math.inf)
        near, at = d2.min(dim=1)
        best[i0:i1] = torch.where(torch.isfinite(near), j0 + at, -1)
    n = best.numel()
    top = torch.where(best >= 0, best, torch.arange(n, device=best.device))
    while not torch.equal(top, top[top]):
        top = top[top]
    label = torch.full((n,), -1, dtype=torch.int64, device=best.device)
    seeds = (best < 0) & seed_like
    point = torch.sort(order[seeds]).values  # clusters are numbered by their seeds' index
    label[seeds] = torch.searchsorted(point, order[seeds])
    out = torch.empty_like(label)
    out[order] = label[top]
    return out


def _scores(case, coords, weights, sizes):
    label = _labels(case, coords, weights, sizes)
    x, w = coords.double(), weights.double()
    k, n = int(label.max()) + 1, label.numel()
    member = torch.nn.functional.one_hot(label[label >= 0], k).double()
    xm, wm = x[:, label >= 0], w[label >= 0]
    size = member.sum(0)
    centroids = (member.T @ xm.T) / size[:, None]
    weighted = (member.T @ (xm * wm).T) / (member.T @ wm)[:, None]
    score = torch.full((n,), math.nan, dtype=torch.float64, device=x.device)
    for i0 in range(0, n, 1024):
        own = label[i0:i0 + 1024]
        d2 = sum((x[d, i0:i0 + 1024, None] - xm[d, None, :]) ** 2 for d in range(case["ndim"]))
        mean = (torch.sqrt(d2) @ member)
        i = torch.arange(own.numel(), device=x.device)
        valid = (own >= 0) & (size[own.clamp(min=0)] >= 2)
        a = mean[i, own.clamp(min=0)] / (size[own.clamp(min=0)] - 1)
        mean = mean / size
        mean[i, own.clamp(min=0)] = math.inf
        b = mean.min(dim=1).values.clamp(max=float(np.finfo(np.float32).max))
        score[i0:i0 + 1024] = torch.where(valid, (b - a) / torch.maximum(a, b), math.nan)
    return {"centroids": centroids, "weighted": weighted, "silhouette": score}


def exact(case, seed):
    if case["where"] != "device" or case["events"] * case["hi"] > 64 * EXACT_POINTS:
        return None
    coords, weights, sizes = _points(case, seed)
    if coords.shape[1] > EXACT_POINTS:
        return None
    if case["call"] == "score":
        return _scores(case, coords, weights, sizes)
    return {"rho": _density(case, coords, weights, sizes), "nearest_higher": None, "is_seed": None,
            "cluster_index": None}
