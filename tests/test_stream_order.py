"""A query on one stream waits for the work of the index's last query on another, also where that one failed after
it had enqueued some (here the order of its queries, in the scratch that both use)."""

import numpy as np
import pytest

import oracle
from cudaexactknn_gb300 import workloads as W

pytestmark = pytest.mark.gpu
gu = pytest.importorskip("gpu_util")

INF = float("inf")


@pytest.mark.parametrize("structure", ["kd", "ball"])
def test_after_a_refused_query(structure):
    import torch
    from cudaexactknn_gb300 import _lib, knn
    rng = np.random.default_rng(1)
    pts, qs = W.uniform(rng, 20000, 3), W.uniform(rng, 9000, 3)
    ix = gu.make_index(structure, pts)
    q = knn.Query(gu.to_dev(qs), len(qs), INF)
    q.ensure_outputs(100)
    ix.batch_knn(q, 100, traversal=1)  # room for the order
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(a):
        torch.cuda._sleep(200_000_000)
    with pytest.raises(_lib.KnnError):  # 256 threads' lists of 128 keys fit no block's shared memory
        ix.batch_knn(q, 100, traversal=1, block_size=256, shmem_tracking=True, sync=False, stream=a)
    enqueued = torch.cuda.Event()
    enqueued.record(a)
    ix.batch_knn(q, 100, traversal=1, sync=False, stream=b)
    b.synchronize()
    assert enqueued.query()
    rows = np.arange(0, len(qs), 50)
    gu.assert_rows_equal(q.r_indexes.cpu().numpy()[rows], q.r_distances.cpu().numpy()[rows],
                         *oracle.bf_knn(pts, qs[rows], 100, fma=True, threads=8))
    torch.cuda.synchronize()
    ix.close()
