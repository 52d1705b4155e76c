"""The warp-per-query tree search: bounds, rows and resumption restated on the CPU, and the kernels
against the oracle at the sizes where a step, a bucket, a scan or a top-k register ends.

Tolerance: none.  Rows are compared as sorted u64 keys with the oracle's fused distances."""

import numpy as np
import pytest

import oracle
from cudaexactknn_gb300 import workloads as W

INF = float("inf")
FAN = 5


# ---- CPU: the control flow ---------------------------------------------------------------------

def _complete_tree(pts, depth, bucket):
    """Slots of a complete median-split tree and its node boxes by (depth, index)."""
    slots = [np.arange(len(pts))]
    for d in range(depth):
        nxt = []
        for s in slots:
            o = s[np.argsort(pts[s, d % pts.shape[1]], kind="stable")]
            nxt += [o[:(len(o) + 1) // 2], o[(len(o) + 1) // 2:]]
        slots = nxt
    assert all(len(s) <= bucket for s in slots)
    boxes = {}
    for d in range(depth + 1):
        for i in range(1 << d):
            ids = np.concatenate(slots[i << (depth - d):(i + 1) << (depth - d)])
            boxes[d, i] = (pts[ids].min(0), pts[ids].max(0)) if len(ids) else None
    return slots, boxes


def _search(q, pts, slots, boxes, depth, k, r2, seed):
    """warp_search of one query: rows of up to 32 bounds, nearest first; with a seed, the least remaining
    bound of a row goes back to its parent and the search resumes past the scanned buckets."""
    def bound(d, i):
        b = boxes[d, i]
        return INF if b is None else float((np.maximum(np.maximum(b[0] - q, q - b[1]), 0) ** 2).sum())
    steps = max(1, -(-depth // FAN))
    lv0 = depth - FAN * (steps - 1)
    top, seen = [], []
    kth = lambda: sorted(top)[k - 1][0] if len(top) >= k else r2
    r, scanned = min(seed, r2), -1.0
    radius = lambda: min(r, kth())

    def expand(row, par):
        d, lv = lv0 + FAN * row, (lv0 if row == 0 else FAN)
        b = {j: bound(d, (par << lv) + j) for j in range(1 << lv)}
        return {j: v for j, v in b.items() if not (row + 1 == steps and v <= scanned)}
    rows, pars = [expand(0, 0)], [0]
    missed = False
    while True:
        row, cur = len(rows) - 1, rows[-1]
        want = [(v, j) for j, v in cur.items() if v <= radius()]
        if not want:
            if row == 0:
                if not r < r2 or not r < kth():
                    return sorted(top)[:k], seen, missed
                scanned, r, missed = r, r2, True
                continue
            rest = min(cur.values(), default=None)
            par = pars.pop()
            rows.pop()
            lv = lv0 if row == 1 else FAN
            if rest is not None:
                rows[-1][par & ((1 << lv) - 1)] = rest
            continue
        _, j = min(want)
        del cur[j]
        child = (pars[-1] << (lv0 if row == 0 else FAN)) + j
        if row + 1 < steps:
            pars.append(child)
            rows.append(expand(row + 1, child))
        else:
            seen.append(child)
            for s in slots[child]:
                d2 = float(((pts[s] - q) ** 2).sum())
                if d2 <= r2:
                    top.append((d2, int(s)))


@pytest.mark.parametrize("depth,n", [(0, 3), (1, 7), (4, 60), (5, 120), (6, 250), (10, 3000), (11, 6000)])
def test_rows_and_resumption_give_brute_force_answers(depth, n):
    rng = np.random.default_rng(depth)
    pts = rng.random((n, 3))
    pts[n // 2:] = pts[n // 2:] * 0.05 + 0.4
    slots, boxes = _complete_tree(pts, depth, 4)
    for q in rng.random((12, 3)):
        d2 = ((pts - q) ** 2).sum(1)
        for k in (1, 5, 8):
            for r2 in (INF, float(np.sort(d2)[min(4, n - 1)])):
                want = sorted((v, i) for i, v in enumerate(d2) if v <= r2)[:k]
                plain, seen_p, _ = _search(q, pts, slots, boxes, depth, k, r2, INF)
                assert [i for _, i in plain] == [i for _, i in want]
                for seed in (0.0, float(np.sort(d2)[min(k - 1, n - 1)]) * 0.5, float(np.sort(d2)[min(k - 1, n - 1)]) * 1.2):
                    got, seen, missed = _search(q, pts, slots, boxes, depth, k, r2, seed)
                    assert [i for _, i in got] == [i for _, i in want]
                    assert len(set(seen)) == len(seen)      # no bucket scanned twice
                    if not missed:
                        assert set(seen) <= set(seen_p)     # a seed that holds only saves


# ---- GPU ---------------------------------------------------------------------------------------

gpu = pytest.mark.gpu


def _gu():
    import gpu_util
    return gpu_util


def _want(pts, qs, k, r2=INF):
    return oracle.bf_knn(pts, qs, k, r2, fma=True, threads=8)


# 32-slot buckets: 1 to 3 of them, one step's 32 (1,024 slots) and one more, two steps and one more.
@gpu
@pytest.mark.parametrize("n", [1, 31, 32, 33, 65, 1024, 1025, 32768, 32769])
@pytest.mark.parametrize("structure", ["kd", "ball"])
def test_steps_and_buckets(structure, n):
    gu = _gu()
    rng = np.random.default_rng(n)
    pts = W.uniform(rng, n, 3)
    pts[n // 2:] = pts[n // 2:] * np.float32(0.02)
    qs = W.uniform(rng, 200, 3)
    for skips in (0, 2, 6):
        ix = gu.make_index(structure, pts, skips)
        for k in (1, 32, 33, 64, 65, 128):
            for r2 in (INF, 1e-3):
                for leaf in (0, 128):
                    gu.assert_rows_equal(*gu.run(ix, qs, k, r2, leaf_scan=leaf), *_want(pts, qs, k, r2),
                                         what=f"{structure} n={n} skips={skips} k={k} r2={r2} leaf={leaf}")
        ix.close()


@gpu
@pytest.mark.parametrize("dims", [1, 4, 5, 16, 17, 33, 65, 128])
@pytest.mark.parametrize("structure", ["kd", "ball"])
def test_dims_seeds_and_resumption(structure, dims):
    """Learned seeds, good, and (margin forced low) too short for every query."""
    from cudaexactknn_gb300 import _lib, knn
    gu = _gu()
    rng = np.random.default_rng(dims)
    pts, centres = W.mixture(rng, 6000, dims, 16, 0.05)
    qs, _ = W.mixture(rng, 500, dims, 16, 0.05, centres)
    ix = gu.make_index(structure, pts, 1)
    ix.train_radius_model(gu.to_dev(qs), 10, steps=50)
    params = ix.export_radius_model()
    for shift in (0.0, -3.0, -30.0):
        p = params.copy()
        p[-1] += shift
        ix.import_radius_model(p, 10)
        for k, r2 in ((10, INF), (10, 0.02 * dims), (40, INF)):
            got = gu.run(ix, qs, k, r2, flags=_lib.QF_LEARNED_RADIUS)
            gu.assert_rows_equal(*got, *_want(pts, qs, k, r2), what=f"{structure} D={dims} shift={shift} k={k} r2={r2}")
    gu.assert_rows_equal(*gu.run(ix, qs, 10), *_want(pts, qs, 10), what=f"{structure} D={dims} unseeded")
    ix.close()


@gpu
@pytest.mark.parametrize("structure", ["kd", "ball"])
def test_captured_queries(structure):
    """A first query inside a stream capture, before anything is built for the index, and a later one."""
    import torch
    from cudaexactknn_gb300 import knn
    gu = _gu()
    rng = np.random.default_rng(4)
    pts, qs = W.uniform(rng, 20000, 3), W.uniform(rng, 700, 3)
    want = _want(pts, qs, 12)
    ix = gu.make_index(structure, pts, 1)
    q = knn.Query(gu.to_dev(qs), len(qs), INF)
    q.ensure_outputs(12)
    for _ in range(2):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            ix.batch_knn(q, 12, sync=False)
        q.r_indexes.fill_(7)
        g.replay()
        torch.cuda.synchronize()
        gu.assert_rows_equal(q.r_indexes.cpu().numpy(), q.r_distances.cpu().numpy(), *want, what="captured")
        gu.assert_rows_equal(*gu.run(ix, qs, 12), *want, what="not captured")
    ix.close()


@gpu
def test_batch_classes_take_a_warp_per_query():
    from cudaexactknn_gb300 import knn
    gu = _gu()
    rng = np.random.default_rng(6)
    items, data = [], []
    for structure, dims, n, nq, k in [("kd", 3, 5, 3, 4), ("kd", 3, 40000, 1000, 4), ("kd", 3, 700, 1, 8), ("kd", 8, 3000, 90, 64),
                                      ("kd", 20, 2000, 33, 100), ("kd", 2, 1, 2, 1), ("ball", 3, 40000, 1000, 4),
                                      ("ball", 3, 9, 2, 8), ("ball", 16, 3000, 90, 64), ("ball", 100, 500, 33, 100)]:
        pts, qs = W.uniform(rng, n, dims), W.uniform(rng, nq, dims)
        data.append((pts, qs, k))
        items.append((gu.make_index(structure, pts, 1), gu.to_dev(qs), k, INF))
    batch = knn.Batch(items)
    for _ in range(2):
        for (pts, qs, k), (idx, dist) in zip(data, batch.run()):
            gu.assert_rows_equal(idx.cpu().numpy(), dist.cpu().numpy(), *_want(pts, qs, k), what=f"{pts.shape} k={k}")
    batch.close()
