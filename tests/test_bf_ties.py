"""Brute force where many points are equally far: the smaller indexes win, whatever a warp has already kept and
whichever warp or block scans them.  Rows are compared as sorted u64 keys: no tolerance."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
gu = pytest.importorskip("gpu_util")

INF = float("inf")


@pytest.mark.parametrize("values", [1, 2, 5])
@pytest.mark.parametrize("dims,n,count,k", [(1, 3000, 40, 32), (3, 40000, 20, 8), (3, 9000, 200, 33), (4, 700, 17, 100),
                                            (8, 30000, 70, 20), (16, 5000, 9, 64), (64, 3000, 600, 20), (100, 2000, 9, 128)])
def test_grid_points(dims, n, count, k, values):
    rng = np.random.default_rng(n + values)
    pts = rng.integers(0, values, (n, dims)).astype(np.float32)
    qs = rng.integers(0, values + 1, (count, dims)).astype(np.float32)
    ix = gu.make_index("bf", pts)
    for r2 in (INF, 0.0, 1.0, 3.0):
        gu.assert_rows_equal(*gu.run(ix, qs, k, r2), *oracle.bf_knn(pts, qs, k, r2, fma=True, threads=8), what=f"r2={r2}")
    ix.close()
