"""Timed cases of the exact-kNN engine: the calls a user of the package makes, at the sizes they come in.

A case is a dict of plain values; ``prepare`` makes on the GPU what a program holds before the call (points,
queries, a built index, a trained radius model, a captured batch), ``run`` is one pass through the public
classes of ``cudaexactknn_gb300.knn``, ``exact`` the same distances in float64 from plain torch.

Kinds of case:

* ``query``   one ``knn`` call on a kept index (brute force, k-d or ball tree; default options, another
              traversal, the learned radius or the tensor-core filter), results on the GPU;
* ``host``    one ``knn_host`` call: pinned host queries in, pinned host rows out;
* ``build``   a tree built over new points, queried once and closed (one-shot use);
* ``batch``   many uneven sets answered by one ``Batch.run``;
* ``train``   one training of an index's radius model (forward, backward, Adam, calibration).
"""

from __future__ import annotations

import math

import torch

from cudaexactknn_gb300 import _lib, knn

INF = float("inf")
OPTS = {  # options of a query by name: keyword arguments of ``knn`` / ``knn_host``
    "default": {},
    "heap": {"heap": True},
    "box": {"traversal": 3, "leaf_scan": 8},
    "learned": {"traversal": 2, "leaf_scan": 16, "flags": _lib.QF_LEARNED_RADIUS},
    "filter": {"flags": _lib.QF_BF16_FILTER},
}
SAMPLES = 65536        # training queries of a learned-radius index
EXACT_PAIRS = 1e11     # most query-point pairs (times dims / 3) that exact() goes through


def _query(name, structure, dims, n, q, k, opts, dist, skips=0, r2=None, kind="query"):
    case = {"kind": kind, "structure": structure, "dims": dims, "n": n, "q": q, "k": k,
            "opts": opts, "dist": dist, "skips": skips, "r2": r2}
    return {"name": name, **case} if name else case


def listed():
    return [
        # A handful of queries against a small table, as an interactive or per-frame caller makes
        # them: all latency.
        _query("bf3_few", "bf", 3, 4096, 16, 8, "default", "uniform"),
        # The brute-force benchmark configuration: 65,536 uniform points, 4,096 queries, k 8, heap
        # tracking.
        _query("bf3_c1", "bf", 3, 65536, 4096, 8, "heap", "uniform"),
        # The k-d tree benchmark configuration (clustered 3-d points, 1,048,576 queries, k 16) as
        # code written against the reference calls it: no option set.
        _query("kd3_default", "kd", 3, 4194304, 1048576, 16, "default", "mixture"),
        # The same with the traversal the engine recommends where there are no training queries.
        _query("kd3_box", "kd", 3, 4194304, 1048576, 16, "box", "mixture"),
        # The same with a trained radius model and the warp-group search: the headline form.
        _query("kd3_learned", "kd", 3, 4194304, 1048576, 16, "learned", "mixture"),
        # The reference's range-limited speed test (N 500,000, Q 10,000, K 5, r2 0.01 D) in 11
        # dimensions, end to end on host buffers.
        _query("kd11_range_host", "kd", 11, 500000, 10000, 5, "default", "uniform", 3, 0.11, "host"),
        # A mid-sized ball tree with default options: data near a 4-d subspace of 16 dimensions.
        _query("ball16_default", "ball", 16, 262144, 65536, 32, "default", "subspace", 1),
        # The ball tree benchmark configuration through the tensor-core filter.
        _query("ball16_filter", "ball", 16, 1048576, 262144, 32, "filter", "subspace", 1),
        # The brute-force embedding-search configuration (128 dimensions, k 100) through the filter.
        _query("bf128_filter", "bf", 128, 1048576, 65536, 100, "filter", "gauss_mix"),
        # One-shot use: a k-d tree over the benchmark's points, 4,096 queries, then closed.
        _query("kd3_build", "kd", 3, 4194304, 4096, 16, "default", "mixture", kind="build"),
        # Uneven independent sets (sizes log-uniform, k from {1, 10, 64}) in one graph launch.
        {"name": "batch_uneven", "kind": "batch", "sets": 24, "lo": 1024, "hi": 262144, "shape": 5},
        # Training the radius model of a k-d tree index.
        {"name": "train_kd3", "kind": "train", "dims": 3, "n": 1048576, "samples": 65536, "k": 16, "steps": 500},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["bf", "bf", "kd", "kd", "kd", "host", "ball", "filter", "filter", "build", "batch", "train"])
    k = rng.choice([1, 5, 8, 10, 16, 20, 32, 50, 64, 100])
    if kind == "bf":
        dims = _log_int(rng, 1, 64)
        n = _log_int(rng, 1000, 300000)
        q = _log_int(rng, 1, max(2, min(20000, int(6e9 / (n * (dims + 8))))))
        return _query(None, "bf", dims, n, q, k, rng.choice(["default", "heap"]), rng.choice(["uniform", "mixture"]))
    if kind == "kd":
        dims = rng.choice([2, 3, 3, 4, 6, 8])
        opts = rng.choice(["default", "box", "learned"])
        k = min(k, 32) if opts == "learned" else k
        n = _log_int(rng, 20000, 2000000 if dims <= 4 else 300000)
        return _query(None, "kd", dims, n, _log_int(rng, 100, n // 4), k, opts,
                      rng.choice(["uniform", "mixture"]) if dims <= 4 else "mixture", rng.choice([0, 0, 1, 3]))
    if kind == "host":
        dims = rng.randint(6, 12)
        structure = rng.choice(["kd", "ball"])
        return _query(None, structure, dims, _log_int(rng, 50000, 500000), _log_int(rng, 100, 10000), 5, "default",
                      "uniform", 3 if structure == "kd" else 1, 0.01 * dims, "host")
    if kind == "ball":
        dims = rng.choice([3, 6, 10, 16, 24])
        return _query(None, "ball", dims, _log_int(rng, 10000, 262144), _log_int(rng, 100, 50000), min(k, 64), "default",
                      "mixture" if dims < 8 else "subspace", rng.choice([1, 2, 3]))
    if kind == "filter":
        dims = rng.choice([16, 20, 32, 50, 64, 96, 128])
        return _query(None, rng.choice(["bf", "ball"]), dims, _log_int(rng, 20000, 600000), _log_int(rng, 500, 50000), k,
                      "filter", "subspace" if dims <= 32 else "gauss_mix", 1)
    if kind == "build":
        dims = rng.choice([2, 3, 5, 8, 16])
        return _query(None, rng.choice(["kd", "ball"]), dims, _log_int(rng, 20000, 3000000 // max(1, dims // 3)),
                      _log_int(rng, 100, 4096), min(k, 32), "default", "mixture", 1, kind="build")
    if kind == "batch":
        return {"kind": "batch", "sets": rng.randint(3, 40), "lo": 1024, "hi": _log_int(rng, 8192, 200000),
                "shape": rng.randrange(1 << 20)}
    return {"kind": "train", "dims": rng.choice([2, 3, 4, 6, 8]), "n": _log_int(rng, 50000, 500000),
            "samples": _log_int(rng, 4000, 60000), "k": min(k, 32), "steps": rng.randint(50, 400)}


# ---- inputs ------------------------------------------------------------------------------------

def _points(gen, dist, dims, *counts):
    """Point sets of one distribution (the same mixture or subspace for every set)."""
    dev = gen.device
    if dist == "uniform":
        return [torch.rand((n, dims), generator=gen, device=dev) for n in counts]
    if dist == "mixture":      # 64 clusters of sigma 0.01 in the unit cube
        centres, sigma = torch.rand((64, dims), generator=gen, device=dev), 0.01
    elif dist == "gauss_mix":  # 256 clusters, centres N(0, 1), sigma 0.3
        centres, sigma = torch.randn((256, dims), generator=gen, device=dev), 0.3
    else:                      # a 4-d linear subspace plus noise
        basis = torch.randn((dims, 4), generator=gen, device=dev, dtype=torch.float64).cpu()
        basis = torch.linalg.qr(basis)[0].float().to(dev)
        return [torch.randn((n, 4), generator=gen, device=dev) @ basis.T +
                0.05 * torch.randn((n, dims), generator=gen, device=dev) for n in counts]
    out = []
    for n in counts:
        which = torch.randint(0, len(centres), (n,), generator=gen, device=dev)
        out.append(centres[which] + sigma * torch.randn((n, dims), generator=gen, device=dev))
    return out


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _r2(case):
    return INF if case["r2"] is None else float(case["r2"])


def _index(case, points):
    if case["structure"] == "bf":
        return knn.BruteForceGpu(points)
    if case["structure"] == "kd":
        return knn.KdTreeGpu(points, depth_skips=case["skips"])
    return knn.BallTreeGpu(points, depth_skips=max(1, case["skips"]))


def _inputs(case, seed):
    return _points(_generator(seed), case["dist"], case["dims"], case["n"], case["q"])


def _batch_shapes(case):
    """(structure, dims, n, queries, k) of each set, from the case alone."""
    import random
    rng = random.Random(case["shape"])
    shapes = []
    for i in range(case["sets"]):
        structure, dims = rng.choice([("kd", 3), ("kd", 3), ("kd", 8), ("ball", 3), ("ball", 16)])
        n = _log_int(rng, case["lo"], case["hi"] if dims == 3 else max(case["lo"], case["hi"] // 8))
        shapes.append((structure, dims, n, max(1, n // 8), rng.choice([1, 10, 64])))
    return shapes


def _batch_inputs(case, seed):
    gen = _generator(seed)
    return [_points(gen, "mixture" if dims < 16 else "subspace", dims, n, q) for _, dims, n, q, _ in _batch_shapes(case)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        items = []
        for (structure, _, _, _, k), (pts, qs) in zip(_batch_shapes(case), _batch_inputs(case, seed)):
            items.append((knn.build_index(structure, pts), qs, k, INF))
        return {"case": case, "batch": knn.Batch(items)}
    if kind == "train":
        pts, samples = _points(_generator(seed), "mixture", case["dims"], case["n"], case["samples"])
        return {"case": case, "index": knn.KdTreeGpu(pts), "samples": samples}
    pts, qs = _inputs(case, seed)
    if kind == "build":
        return {"case": case, "points": pts, "queries": qs}
    state = {"case": case, "index": _index(case, pts), "queries": qs}
    if case["opts"] == "learned":
        # The program trains on a sample of its own queries.
        sample = qs if len(qs) <= SAMPLES else qs[torch.randperm(len(qs), generator=_generator(seed + 1), device=qs.device)[:SAMPLES]]
        state["index"].train_radius_model(sample, case["k"], steps=1000)
    if kind == "host":
        state["queries"] = qs.cpu().pin_memory()
        state["out_idx"] = torch.empty((case["q"], case["k"]), dtype=torch.int32, pin_memory=True)
        state["out_dist"] = torch.empty((case["q"], case["k"]), dtype=torch.float32, pin_memory=True)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        return state["batch"].run()
    if kind == "train":
        report = state["index"].train_radius_model(state["samples"], case["k"], steps=case["steps"])
        return {"params": state["index"].export_radius_model(), "loss": report.final_batch_loss, "rmse": report.rmse,
                "margin": report.margin, "coverage": report.coverage}
    if kind == "build":
        index = _index(case, state["points"])
        out = index.knn(state["queries"], case["k"], _r2(case), **OPTS[case["opts"]])
        index.close()
        return out
    if kind == "host":
        return state["index"].knn_host(state["queries"], case["k"], _r2(case), state["out_idx"], state["out_dist"],
                                       **OPTS[case["opts"]])
    return state["index"].knn(state["queries"], case["k"], _r2(case), **OPTS[case["opts"]])


# ---- what a pass cannot do without, and its exact distances --------------------------------------

def _query_work(dims, n, q, k):
    """Points, queries and rows once; the k distances of every row."""
    return 4.0 * dims * (n + q) + 8.0 * q * k, 3.0 * dims * q * min(k, n)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        parts = [_query_work(dims, n, q, k) for _, dims, n, q, k in _batch_shapes(case)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    if kind == "train":
        feats = case["dims"] + 64
        batch = min(1024, case["samples"])
        macs = 64 * feats + 64 * 64 + 64
        b, f = _query_work(case["dims"], case["n"], case["samples"], case["k"])
        return {"bytes": b + 4.0 * case["steps"] * batch * (case["dims"] + 1),
                "flops": f + 6.0 * macs * batch * case["steps"]}
    b, f = _query_work(case["dims"], case["n"], case["q"], case["k"])
    if case["structure"] == "bf" and case["opts"] != "filter":
        f = 3.0 * case["dims"] * case["n"] * case["q"]  # brute force is every pair
    return {"bytes": b, "flops": f}


def _rows64(points, queries, k, r2):
    """The k smallest squared distances of every query in float64, ascending; r2 where fewer lie within it."""
    p, q = points.double(), queries.double()
    n, kk = len(p), min(k, len(p))
    out = torch.full((len(q), k), r2, dtype=torch.float64, device=q.device)
    step = max(1, int(4e8 / n))
    for i in range(0, len(q), step):
        c = q[i:i + step]
        d = torch.zeros((len(c), n), dtype=torch.float64, device=q.device)
        for j in range(p.shape[1]):
            t = c[:, j, None] - p[None, :, j]
            d.addcmul_(t, t)
        out[i:i + step, :kk] = torch.clamp(torch.topk(d, kk, dim=1, largest=False, sorted=True)[0], max=r2)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return None
    if kind == "batch":
        shapes = _batch_shapes(case)
        if sum(dims * n * q for _, dims, n, q, _ in shapes) > EXACT_PAIRS:
            return None
        return [(None, _rows64(pts, qs, k, INF)) for (_, _, _, _, k), (pts, qs) in zip(shapes, _batch_inputs(case, seed))]
    if case["n"] * case["q"] * max(1.0, case["dims"] / 3) > EXACT_PAIRS:
        return None
    pts, qs = _inputs(case, seed)
    return (None, _rows64(pts, qs, case["k"], _r2(case)))
