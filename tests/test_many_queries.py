"""Batches of so many queries, of so few dims and neighbours, that each query gets a thread (in locality order)
instead of a warp: the rows are the oracle's as everywhere, on both sides of the line, for queries near and far
from the points, per-query radii, equal points, and inside a stream capture with and without room for the order.
Rows are compared as sorted u64 keys: no tolerance."""

import numpy as np
import pytest

import oracle
from cudaexactknn_gb300 import workloads as W

pytestmark = pytest.mark.gpu
gu = pytest.importorskip("gpu_util")

INF = float("inf")


def _case(dims, n, count):
    rng = np.random.default_rng(dims * 7 + n)
    pts, centres = W.mixture(rng, n, dims, 16, 0.01)
    pts[n // 2:n // 2 + 20] = pts[:20] if n >= 60 else pts[n // 2:n // 2 + 20]  # equal points
    near, _ = W.mixture(rng, count, dims, 16, 0.01, centres)
    near[::5] = (W.uniform(rng, len(near[::5]), dims) - np.float32(0.5)) * np.float32(40)  # far
    near[::7] = pts[rng.integers(0, n, len(near[::7]))]
    return pts, near, np.unique(np.concatenate([np.arange(0, count, count // 200), [1, count - 1]]))


@pytest.mark.parametrize("structure,dims,n,count,ks,skips", [
    ("kd", 1, 5000, 250000, (1, 8, 9), 0), ("kd", 1, 3, 500000, (9, 16), 0), ("kd", 1, 20000, 500000, (16,), 4),
    ("kd", 2, 3000, 800000, (1, 4, 5), 0), ("kd", 2, 3000, 800000, (4,), 7), ("kd", 3, 900, 1000000, (1, 2, 3), 2),
    ("ball", 1, 5000, 250000, (1, 8, 9), 1), ("ball", 1, 700, 500000, (16,), 3), ("ball", 2, 9000, 500000, (1, 2, 3), 1),
    ("ball", 3, 9000, 500000, (2,), 5), ("ball", 4, 9000, 1000000, (1, 8, 9), 1), ("ball", 2, 1, 1000000, (8,), 1),
    ("kd", 24, 320, 200000, (1, 16, 17), 0), ("kd", 100, 320, 200000, (5,), 3), ("kd", 4, 64, 200000, (4, 5), 1), ("kd", 12, 64, 1000000, (16,), 0),
    ("ball", 3, 64, 200000, (4, 5), 1), ("ball", 4, 1024, 1000000, (16,), 2)])
def test_rows(structure, dims, n, count, ks, skips):
    pts, qs, rows = _case(dims, n, count)
    dq = gu.to_dev(qs)
    ix = gu.make_index(structure, pts, skips)
    for k in ks:
        for r2 in (INF, 1e-3):
            idx, dist = ix.knn(dq, k, r2)
            want = oracle.bf_knn(pts, qs[rows], k, r2, fma=True, threads=8)
            gu.assert_rows_equal(idx.cpu().numpy()[rows], dist.cpu().numpy()[rows], *want, what=f"k={k} r2={r2}")
    # One query fewer than the line, and the caller's order: a warp each, the same rows everywhere.
    from cudaexactknn_gb300 import _lib
    k = ks[0]
    idx, dist = ix.knn(dq, k)
    for other in (ix.knn(dq[:-1].contiguous(), k), ix.knn(dq, k, flags=_lib.QF_KEEP_ORDER)):
        m = len(other[0])
        assert (other[0] == idx[:m]).all() and (other[1] == dist[:m]).all()
    ix.close()


@pytest.mark.parametrize("structure", ["kd", "ball"])
def test_radii_and_counters(structure):
    from cudaexactknn_gb300 import knn
    pts, qs, rows = _case(1, 4000, 260000)
    ix = gu.make_index(structure, pts)
    radii = np.tile(np.array([0.0, 1e-6, 1e-2, INF], np.float32), len(qs))[:len(qs)]
    q = knn.Query(gu.to_dev(qs), len(qs), 0.0)
    idx, dist = ix.batch_knn_radii(q, gu.to_dev(radii), 6)
    for r in rows[:60]:
        want = oracle.bf_knn(pts, qs[r:r + 1], 6, float(radii[r]), fma=True, threads=8)
        gu.assert_rows_equal(idx[r:r + 1].cpu().numpy(), dist[r:r + 1].cpu().numpy(), *want, what=f"radius {radii[r]}")
    c = ix.stats(knn.Query(gu.to_dev(qs), len(qs), INF), 6)
    assert c.points_scanned >= 6 * len(qs) and c.leaves_visited > 0 and c.fallback_queries == 0
    ix.close()


@pytest.mark.parametrize("structure", ["kd", "ball"])
def test_captured(structure):
    import torch
    from cudaexactknn_gb300 import knn
    pts, qs, rows = _case(1, 4000, 260000)
    want = oracle.bf_knn(pts, qs[rows], 5, fma=True, threads=8)
    ix = gu.make_index(structure, pts)
    q = knn.Query(gu.to_dev(qs), len(qs), INF)
    q.ensure_outputs(5)
    for _ in range(2):  # before any query made room for an order, and after
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            ix.batch_knn(q, 5, sync=False)
        q.r_indexes.fill_(7)
        g.replay()
        torch.cuda.synchronize()
        gu.assert_rows_equal(q.r_indexes.cpu().numpy()[rows], q.r_distances.cpu().numpy()[rows], *want, what="captured")
        ix.batch_knn(q, 5)
        gu.assert_rows_equal(q.r_indexes.cpu().numpy()[rows], q.r_distances.cpu().numpy()[rows], *want, what="not captured")
    ix.close()
