"""A query that is refused (a block's shared memory cannot hold what the options ask for) leaves nothing behind: the
next query answers."""

import numpy as np
import pytest

import oracle
from cudaexactknn_gb300 import workloads as W

pytestmark = pytest.mark.gpu
gu = pytest.importorskip("gpu_util")


@pytest.mark.parametrize("structure,traversal", [("kd", 1), ("ball", 1), ("kd", 0), ("ball", 0), ("bf", 0)])
def test_the_next_query_answers(structure, traversal):
    from cudaexactknn_gb300 import _lib
    rng = np.random.default_rng(3)
    pts, qs = W.uniform(rng, 5000, 3), W.uniform(rng, 300, 3)
    want = oracle.bf_knn(pts, qs, 100, fma=True, threads=8)
    ix = gu.make_index(structure, pts)
    for _ in range(2):
        with pytest.raises(_lib.KnnError):  # 256 threads' lists of 128 keys: 256 KB
            gu.run(ix, qs, 100, traversal=traversal, block_size=256, shmem_tracking=True)
        gu.assert_rows_equal(*gu.run(ix, qs, 100, traversal=traversal), *want)
    ix.close()
