"""Brute force's thread-per-query form at the sizes where it takes over from the warps and at its own edges: the
places min(k, n) leaves empty, odd numbers of points, tiles and splits of the points, a last block of few
queries, per-query radii, and the allocation-free entry point.  Rows are compared as sorted u64 keys with the
oracle's fused distances: no tolerance."""

import ctypes

import numpy as np
import pytest

import oracle
from cudaexactknn_gb300 import workloads as W

pytestmark = pytest.mark.gpu
gu = pytest.importorskip("gpu_util")

INF = float("inf")


def _noalloc(pts, qs, k, r2):
    import torch
    from cudaexactknn_gb300 import _lib
    p, q = gu.to_dev(pts), gu.to_dev(qs)
    idx = torch.full((len(qs), k), 7, dtype=torch.int32, device=p.device)
    dist = torch.full((len(qs), k), 7.0, device=p.device)
    _lib.check(_lib.load().knn_bf_query_noalloc(p.data_ptr(), len(pts), pts.shape[1], q.data_ptr(), len(qs), ctypes.c_float(r2),
                                                k, idx.data_ptr(), dist.data_ptr(), None))
    torch.cuda.synchronize()
    return idx.cpu().numpy(), dist.cpu().numpy()


@pytest.mark.parametrize("dims", [1, 3, 4, 5, 16, 20, 64, 100])
@pytest.mark.parametrize("n,count,k", [
    (1, 1, 1), (1, 3, 32), (7, 129, 8), (8, 64, 8), (9, 1000, 9), (16, 63, 32), (17, 63, 17), (17, 64, 17), (32, 130, 20),
    (33, 130, 32), (64, 64, 8), (64, 100, 16), (65, 100, 16), (128, 65, 3), (129, 65, 3), (200, 12287, 5), (200, 12289, 5),
    (100, 12300, 12), (61, 12300, 31), (512, 65600, 1), (1023, 12300, 8)])
def test_rows(dims, n, count, k):
    rng = np.random.default_rng(n * 131 + count + dims)
    pts, qs = W.uniform(rng, n, dims), W.uniform(rng, count, dims)
    pts[n // 2:] = pts[:n - n // 2]  # equal distances: the smaller index wins
    rows = np.unique(np.concatenate([np.arange(min(count, 40)), np.arange(0, count, max(1, count // 150)),
                                     np.arange(max(0, count - 40), count)]))
    ix = gu.make_index("bf", pts)
    for r2 in (INF, 0.05 * dims):
        want = oracle.bf_knn(pts, qs[rows], k, r2, fma=True, threads=8)
        for got in (gu.run(ix, qs, k, r2), _noalloc(pts, qs, k, r2)):
            gu.assert_rows_equal(got[0][rows], got[1][rows], *want, what=f"r2={r2}")
            gu.assert_sorted_rows(*got)
    ix.close()


# Points split over blocks: a last chunk of one point, of a whole tile, and many chunks.
@pytest.mark.parametrize("dims,n,count,k", [(20, 1025, 12300, 8), (20, 3 * 1024 + 256, 6000, 3), (33, 20001, 700, 8),
                                            (100, 20001, 160, 16), (128, 1024, 4000, 32), (8, 16384, 9000, 8),
                                            (64, 70000, 70, 2)])
def test_splits(dims, n, count, k):
    import torch
    from cudaexactknn_gb300 import knn
    rng = np.random.default_rng(n)
    pts, qs = W.uniform(rng, n, dims), W.uniform(rng, count, dims)
    rows = np.arange(0, count, max(1, count // 60))
    want = oracle.bf_knn(pts, qs[rows], k, fma=True, threads=8)
    ix = gu.make_index("bf", pts)
    got = gu.run(ix, qs, k)
    gu.assert_rows_equal(got[0][rows], got[1][rows], *want)
    got = _noalloc(pts, qs, k, INF)
    gu.assert_rows_equal(got[0][rows], got[1][rows], *want, what="noalloc")
    # A radius per query: none, one that holds some of its k, one that holds all.
    radii = np.tile(np.array([0.0, want[1][:, k // 2].mean(), INF], np.float32), count)[:count]
    q = knn.Query(gu.to_dev(qs), count, 0.0)
    ri, rd = ix.batch_knn_radii(q, gu.to_dev(radii), k)
    for i, r in enumerate(rows):
        w = oracle.bf_knn(pts, qs[r:r + 1], k, float(radii[r]), fma=True, threads=8)
        gu.assert_rows_equal(ri[r:r + 1].cpu().numpy(), rd[r:r + 1].cpu().numpy(), *w, what=f"radius {radii[r]}")
    torch.cuda.synchronize()
    ix.close()


def test_more_places_than_points():
    rng = np.random.default_rng(2)
    pts, qs = W.uniform(rng, 11, 64), W.uniform(rng, 16400, 64)
    for k in (40, 128):
        got = gu.run(gu.make_index("bf", pts), qs, k, 6.0)
        rows = np.arange(0, len(qs), 101)
        gu.assert_rows_equal(got[0][rows], got[1][rows], *oracle.bf_knn(pts, qs[rows], k, 6.0, fma=True, threads=8))
