"""The k-d tree's node boxes come with the tree, reach the buckets that are searched, and are complete
before anything reads them: batch graphs, training and captured queries run on streams that do not wait
for the stream of the index's first query."""

import numpy as np
import pytest

import oracle
from cudaexactknn_gb300 import workloads as W

pytestmark = pytest.mark.gpu
gu = pytest.importorskip("gpu_util")

INF = float("inf")
DELAY = 200_000_000  # cycles a stream is kept busy: about 0.1 s


def _case(dims, n=60000, q=3000, k=10):
    rng = np.random.default_rng(dims)
    pts = W.uniform(rng, n, dims)
    qs = W.uniform(rng, q, dims)
    return pts, qs, oracle.bf_knn(pts, qs, k, fma=True, threads=8)


def _delayed_first_query(ix, qs, k, stream):
    """The index's first query, enqueued behind work that keeps its stream busy."""
    import torch
    from cudaexactknn_gb300 import knn
    q = knn.Query(gu.to_dev(qs), len(qs), INF)
    q.ensure_outputs(k)
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(DELAY)
    ix.batch_knn(q, k, sync=False, stream=stream)
    return q


@pytest.mark.parametrize("dims", [3, 11, 40])
def test_batch_beside_the_first_query(dims):
    import torch
    from cudaexactknn_gb300 import knn
    pts, qs, want = _case(dims)
    ix = gu.make_index("kd", pts)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    dq = gu.to_dev(qs)
    q = _delayed_first_query(ix, qs, 10, a)
    batch = knn.Batch([(ix, dq, 10, INF)], stream=b)
    (idx, dist), = batch.run(stream=b)
    got = idx.cpu().numpy(), dist.cpu().numpy()
    torch.cuda.synchronize()
    gu.assert_rows_equal(*got, *want, what="batch on another stream")
    gu.assert_rows_equal(q.r_indexes.cpu().numpy(), q.r_distances.cpu().numpy(), *want, what="first query")
    batch.close()
    ix.close()


@pytest.mark.parametrize("dims", [3, 40])
def test_batch_created_and_run_on_different_streams(dims):
    import torch
    from cudaexactknn_gb300 import knn
    pts, qs, want = _case(dims)
    ix = gu.make_index("kd", pts)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    dq = gu.to_dev(qs)
    torch.cuda.synchronize()
    with torch.cuda.stream(a):
        torch.cuda._sleep(DELAY)
    batch = knn.Batch([(ix, dq, 10, INF)], stream=a)
    (idx, dist), = batch.run(stream=b)
    gu.assert_rows_equal(idx.cpu().numpy(), dist.cpu().numpy(), *want, what="run on another stream")
    torch.cuda.synchronize()
    batch.close()
    ix.close()


def test_capture_on_another_stream():
    import torch
    from cudaexactknn_gb300 import knn
    pts, qs, want = _case(3)
    ix = gu.make_index("kd", pts)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    c = knn.Query(gu.to_dev(qs), len(qs), INF)
    c.ensure_outputs(10)
    _delayed_first_query(ix, qs, 10, a)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(b):
        graph.capture_begin(capture_error_mode="thread_local")
        ix.batch_knn(c, 10, sync=False, stream=b)
        graph.capture_end()
        graph.replay()
    b.synchronize()
    gu.assert_rows_equal(c.r_indexes.cpu().numpy(), c.r_distances.cpu().numpy(), *want, what="captured beside the build")
    torch.cuda.synchronize()
    ix.close()


def test_training_beside_the_first_query():
    """Training's targets are the samples' exact k-th distances: the same model as on an idle index."""
    import torch
    pts, qs, _ = _case(3)
    models = []
    for delayed in (False, True):
        ix = gu.make_index("kd", pts)
        a, b = torch.cuda.Stream(), torch.cuda.Stream()
        samples = gu.to_dev(qs)
        if delayed:
            _delayed_first_query(ix, qs, 10, a)
        else:
            torch.cuda.synchronize()
        ix.train_radius_model(samples, 10, steps=20, stream=b)
        models.append(ix.export_radius_model())
        torch.cuda.synchronize()
        ix.close()
    np.testing.assert_array_equal(models[0].view(np.uint32), models[1].view(np.uint32))


@pytest.mark.parametrize("dims", [3, 12, 40])
def test_boxes_reach_the_buckets_that_are_searched(dims):
    """An index holds its tree and the boxes of subtrees of 32 slots (16 beyond 8 dims), no deeper, from its
    creation or from its saved form on; the warp-group search's smaller ones come with that search's first
    query.  device_bytes counts all of them."""
    from cudaexactknn_gb300 import knn
    pts, qs, want = _case(dims, n=60000, q=50)
    made = gu.make_index("kd", pts)
    info = made.info()
    row = 4 if dims < 4 else {12: 16, 40: 64}[dims]
    tree = 4 * info.node_count + 4 * (info.node_count + 1) * info.leaf_slots * (4 if dims < 4 else row + 4)
    box = ((2 << (info.node_depth - (5 if dims <= 8 else 4))) - 1) * 2 * 4 * row
    for ix in (made, knn.load_index(made.serialize())):
        assert ix.info().device_bytes == tree + box
        gu.assert_rows_equal(*gu.run(ix, qs, 10), *want)
        assert ix.info().device_bytes == tree + box
        if dims <= 16:
            for _ in range(2):
                gu.assert_rows_equal(*gu.run(ix, qs, 10, traversal=2), *want)
                assert ix.info().device_bytes > tree + 3 * box
            gu.assert_rows_equal(*gu.run(ix, qs, 10), *want)
        ix.close()


# A node's slots over fewer lanes than a warp, one each, and several; dimensions over the lanes beyond 16.
@pytest.mark.parametrize("dims", [1, 3, 9, 16, 17, 100])
@pytest.mark.parametrize("n,skips", [(1, 0), (2, 1), (17, 2), (33, 5), (1000, 0), (1000, 4), (5000, 7), (3000, 30),
                                     (513, 9), (1000, 9)])
def test_boxes_of_every_bucket_size(dims, n, skips):
    rng = np.random.default_rng(n + dims)
    pts = W.uniform(rng, n, dims) - np.float32(0.5)  # both signs: padding's zeros lie inside
    qs = (W.uniform(rng, 40, dims) - np.float32(0.5)) * np.float32(3)
    want = oracle.bf_knn(pts, qs, 5, fma=True, threads=8)
    ix = gu.make_index("kd", pts, skips)
    for traversal in (0, 2, 0) if dims <= 16 else (0,):
        gu.assert_rows_equal(*gu.run(ix, qs, 5, traversal=traversal), *want, what=f"traversal {traversal}")
    ix.close()
