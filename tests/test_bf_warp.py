"""The brute-force kernel where its tiles, steps, parts, splits, buffers and top-k registers end, against
the oracle.  Tolerance: none (rows compared as sorted u64 keys)."""

import numpy as np
import pytest

import oracle
from cudaexactknn_gb300 import workloads as W

pytestmark = pytest.mark.gpu
gu = pytest.importorskip("gpu_util")

INF = float("inf")


def _check(pts, qs, k, r2=INF, what=""):
    ix = gu.make_index("bf", pts)
    want = oracle.bf_knn(pts, qs, k, r2, fma=True, threads=8)
    gu.assert_rows_equal(*gu.run(ix, qs, k, r2), *want, what=what)
    ix.close()


# Tiles hold 512 rows (up to 4 dims), 256 (to 64) or 128; a step 32; a warp 8, 4 or 2 queries.
@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, 511, 513, 1025, 20000])
@pytest.mark.parametrize("dims", [3, 4, 5, 64, 128])
def test_tiles_and_registers(n, dims):
    rng = np.random.default_rng(n + dims)
    pts = W.uniform(rng, n, dims)
    for q, k in ((1, 1), (9, 32), (5, 33), (17, 64), (3, 65), (70, 128)):
        qs = W.uniform(rng, q, dims)
        _check(pts, qs, k, INF, f"n={n} D={dims} q={q} k={k}")
        _check(pts, qs, k, 0.05 * dims, f"n={n} D={dims} q={q} k={k} radius")


# Few queries (parts and splits), as many groups as warps, more (four rows a lane beyond 4 dims).
@pytest.mark.parametrize("q", [1, 2, 63, 64, 65, 700])
@pytest.mark.parametrize("dims,k", [(2, 10), (8, 10), (8, 40), (33, 100)])
def test_shares(q, dims, k):
    rng = np.random.default_rng(q)
    _check(W.uniform(rng, 30000, dims), W.uniform(rng, q, dims), k, INF, f"q={q} D={dims} k={k}")


@pytest.mark.parametrize("dims", [3, 16])
@pytest.mark.parametrize("k", [5, 50, 128])
def test_full_buffers(dims, k):
    """Every point within the bound: equal points (ties by index), and points that come nearer in order, so
    that each tile holds nothing but new neighbours."""
    qs = np.zeros((20, dims), np.float32)
    _check(np.ones((5000, dims), np.float32), qs, k, INF, "equal")
    near = np.linspace(3.0, 0.1, 20000, dtype=np.float32)[:, None] * np.ones((1, dims), np.float32)
    _check(near, qs, k, INF, "ever nearer")
    _check(near[::-1].copy(), qs, k, INF, "ever farther")


@pytest.mark.parametrize("dims,k", [(3, 8), (4, 100), (7, 40), (100, 20)])
def test_allocation_free_form(dims, k):
    import torch
    from cudaexactknn_gb300 import _lib
    rng = np.random.default_rng(dims)
    for n, q in ((5, 3), (9000, 65), (70000, 4)):
        pts, qs = W.uniform(rng, n, dims), W.uniform(rng, q, dims)
        tp, tq = gu.to_dev(pts), gu.to_dev(qs)
        idx = torch.empty((q, k), dtype=torch.int32, device="cuda")
        dist = torch.empty((q, k), dtype=torch.float32, device="cuda")
        _lib.check(_lib.load().knn_bf_query_noalloc(tp.data_ptr(), n, dims, tq.data_ptr(), q, 2.0, k, idx.data_ptr(),
                                                    dist.data_ptr(), torch.cuda.current_stream().cuda_stream))
        gu.assert_rows_equal(idx.cpu().numpy(), dist.cpu().numpy(), *oracle.bf_knn(pts, qs, k, 2.0, fma=True, threads=8),
                             what=f"n={n} q={q} D={dims} k={k}")
