"""The filter's landmark layout with cells of fewer than k points: their queries are assigned to the nearest
landmark whose cell holds k.  Exact rows (no tolerance), and no query tile left scanning the whole table."""

import numpy as np
import pytest

import oracle
from cudaexactknn_gb300 import workloads as W

pytestmark = pytest.mark.gpu
gu = pytest.importorskip("gpu_util")

INF = float("inf")


def _data(dims, n, rng):
    """Clusters, with a lone far point at each position that the layout takes a landmark from."""
    pts, centres = W.gauss_mix(rng, n, dims, 24, 0.3)
    cells = max(1, min(2048, n // 1024))
    at = (np.arange(cells, dtype=np.uint64) * n // cells).astype(np.int64)
    pts[at[::2]] += rng.standard_normal((len(at[::2]), dims)).astype(np.float32) * 2
    qs, _ = W.gauss_mix(rng, 700, dims, 24, 0.3, centres)
    qs[:20] = pts[at[::2]][np.arange(20) % len(at[::2])] + np.float32(0.01)
    return pts, qs


@pytest.mark.parametrize("dims", [40, 128])
@pytest.mark.parametrize("k", [1, 2, 40, 100])
def test_queries_near_lone_landmarks(dims, k):
    from cudaexactknn_gb300 import _lib
    rng = np.random.default_rng(dims + k)
    pts, qs = _data(dims, 30000, rng)
    ix = gu.make_index("bf", pts)
    got = gu.run(ix, qs, k, flags=_lib.QF_BF16_FILTER)
    gu.assert_rows_equal(*got, *oracle.bf_knn(pts, qs, k, fma=True, threads=8), what=f"D={dims} k={k}")
    ix.close()


@pytest.mark.parametrize("n,k", [(90, 100), (600, 128), (1300, 128)])
def test_no_cell_holds_k_points(n, k):
    from cudaexactknn_gb300 import _lib
    rng = np.random.default_rng(n)
    pts, _ = W.gauss_mix(rng, n, 48, 300, 0.01)
    qs, _ = W.gauss_mix(rng, 200, 48, 300, 0.01)
    ix = gu.make_index("bf", pts)
    got = gu.run(ix, qs, k, flags=_lib.QF_BF16_FILTER)
    gu.assert_rows_equal(*got, *oracle.bf_knn(pts, qs, k, fma=True, threads=8), what=f"n={n} k={k}")
    ix.close()
