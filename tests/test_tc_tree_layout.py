"""The filter's tree layout cuts along the widest dimension: points wide in one dimension only, in any of them, at
sizes whose last tile and last warp are full, ragged and nearly empty.

Rows: exact (no tolerance).  Tiles scanned, derived: 500 sorted queries are four tiles of at most 128, each over at
most a quarter of the ~79 point tiles and one more; a query's bound reaches at most |x| / 32 around it (16-bit rows:
2^-10 of |x|^2 in the squared distance), 3 tiles, and lies in its tile and the next: 4 x (21 + 2 x 4) = 116.  A cut
along any other dimension separates nothing, and all 316 are scanned: half of that is the line."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
gu = pytest.importorskip("gpu_util")


@pytest.mark.parametrize("n", [20000, 19968, 19969, 20031])
@pytest.mark.parametrize("dims,wide", [(16, 0), (16, 15), (17, 16), (32, 7), (32, 31)])
def test_widest_dimension(dims, wide, n):
    from cudaexactknn_gb300 import _lib, knn
    rng = np.random.default_rng(n + dims)
    pts = (rng.random((n, dims)) * 1e-3).astype(np.float32)
    qs = (rng.random((500, dims)) * 1e-3).astype(np.float32)
    pts[:, wide] = rng.random(n) - 0.5
    qs[:, wide] = rng.random(500) - 0.5
    ix = gu.make_index("bf", pts)
    want = oracle.bf_knn(pts, qs, 5, fma=True, threads=8)
    gu.assert_rows_equal(*gu.run(ix, qs, 5, flags=_lib.QF_BF16_FILTER), *want, what=f"D={dims} n={n}")
    c = ix.stats(knn.Query(gu.to_dev(qs), 500, float("inf")), 5, flags=_lib.QF_BF16_FILTER)
    assert 0 < c.leaves_visited <= 158
    ix.close()
