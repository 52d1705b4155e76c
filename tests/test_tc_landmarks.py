"""The filter's landmark layout puts every point in the cell of its nearest landmark: separated clusters of 1,024
contiguous points, so that each has one of the landmarks (every 1,024th point), where the last warp and block of
rows are full, ragged and of one row, and the dimensions fill their padding or not.

Rows: exact (no tolerance).  Tiles scanned, derived: 500 queries sorted by cell are four tiles of at most 128; each
meets the cells it spans, and its four tiles' spans of the 40 cells share at most three: 43 cells of at most 5
tiles (one padded) are 215, and one cell for the points past the last cluster makes 220.  Points in wrong cells
leave no cell a radius that prunes: 4 x 160 and more are scanned, and half of that is the line."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
gu = pytest.importorskip("gpu_util")


@pytest.mark.parametrize("extra", [0, 1, 33, 127])
@pytest.mark.parametrize("dims", [33, 64, 65, 128])
def test_nearest_landmark(dims, extra):
    from cudaexactknn_gb300 import _lib, knn
    rng = np.random.default_rng(dims + extra)
    centres = rng.standard_normal((40, dims)) * 10
    which = np.concatenate([np.repeat(np.arange(40), 1024), np.full(extra, 39)])
    pts = (centres[which] + 0.1 * rng.standard_normal((len(which), dims))).astype(np.float32)
    qs = (centres[rng.integers(0, 40, 500)] + 0.1 * rng.standard_normal((500, dims))).astype(np.float32)
    ix = gu.make_index("bf", pts)
    want = oracle.bf_knn(pts, qs, 5, fma=True, threads=8)
    gu.assert_rows_equal(*gu.run(ix, qs, 5, flags=_lib.QF_BF16_FILTER), *want, what=f"D={dims} extra={extra}")
    c = ix.stats(knn.Query(gu.to_dev(qs), 500, float("inf")), 5, flags=_lib.QF_BF16_FILTER)
    assert 0 < c.leaves_visited <= 320
    ix.close()
