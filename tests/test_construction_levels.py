"""Tree construction where its stages meet: subtrees of at most 4,096 points (fewer with more than 16 orders)
finished by one block, partition words of 32 positions and tiles of 2,048, the scan past 4,096 tiles, sort
blocks of 4,096 pairs.  The search with splitting planes (traversal 1) and the one with node boxes or balls
must both equal the oracle's brute force (no tolerance), which no wrong split or misplaced point survives."""

import numpy as np
import pytest

import oracle
from cudaexactknn_gb300 import workloads as W

pytestmark = pytest.mark.gpu
gu = pytest.importorskip("gpu_util")


def _check(structure, pts, qs, k, skips, aux=None):
    ix = gu.make_index(structure, pts, skips, aux)
    want = oracle.bf_knn(pts, qs, k, fma=True, threads=8)
    for traversal in (0, 1):
        gu.assert_rows_equal(*gu.run(ix, qs, k, traversal=traversal), *want,
                             what=f"{structure} n={len(pts)} D={pts.shape[1]} skips={skips} aux={aux} traversal={traversal}")
    ix.close()


@pytest.mark.parametrize("n", [2, 31, 2047, 2049, 4095, 4096, 4097, 8192, 8193, 16411])
@pytest.mark.parametrize("dims,aux", [(1, 1), (3, 3), (4, 2), (16, 16), (17, 17), (128, 128)])
def test_kd_subtrees(n, dims, aux):
    rng = np.random.default_rng(n + dims)
    pts = W.uniform(rng, n, dims)
    pts[n // 3:n // 2] = pts[0]  # equal coordinates: stable order everywhere
    for skips in (0, 2):
        _check("kd", pts, W.uniform(rng, 40, dims), 5, skips, aux)


@pytest.mark.parametrize("n", [33, 2049, 4097, 40000])
def test_ball_partitions(n):
    rng = np.random.default_rng(n)
    _check("ball", W.uniform(rng, n, 5), W.uniform(rng, 40, 5), 5, 1)


def test_partition_past_the_direct_tiles():
    rng = np.random.default_rng(3)
    n = 4096 * 2048 + 777
    _check("kd", W.uniform(rng, n, 2), W.uniform(rng, 24, 2), 4, 0)


@pytest.mark.parametrize("kind", ["equal", "descending", "two values"])
def test_sorted_and_equal_keys(kind):
    """Digits that fill one bucket, and orders that a pass reverses."""
    rng = np.random.default_rng(5)
    n = 13001
    pts = {"equal": np.full((n, 3), 0.5, np.float32),
           "descending": np.linspace(1.0, -1.0, n, dtype=np.float32)[:, None].repeat(3, 1),
           "two values": (rng.random((n, 3)) < 0.5).astype(np.float32)}[kind]
    _check("kd", np.ascontiguousarray(pts), W.uniform(rng, 20, 3), 8, 0)
    _check("ball", np.ascontiguousarray(pts), W.uniform(rng, 20, 3), 8, 1)
