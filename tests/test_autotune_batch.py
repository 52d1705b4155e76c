"""Autotuning where the filter and the structure's own search meet again on more of the batch than the sample: a
batch of at least twice the queries a sample takes (131,072 k-d, 32,768 ball, 8,192 brute force), plain and with
a radius model, and the batch API's class of such a set.  Exact integers and distance bits: no tolerance."""

import numpy as np
import pytest

import oracle
from cudaexactknn_gb300 import workloads as W

pytestmark = pytest.mark.gpu
gu = pytest.importorskip("gpu_util")


@pytest.mark.parametrize("structure,dims,count", [("ball", 16, 65536), ("kd", 16, 262200), ("bf", 16, 17000),
                                                  ("ball", 17, 65535)])
def test_finalists(structure, dims, count):
    from cudaexactknn_gb300 import _lib, knn
    rng = np.random.default_rng(count)
    pts, basis = W.subspace(rng, 1500, dims, 4, 0.05)
    qs, _ = W.subspace(rng, count, dims, 4, 0.05, basis)
    want = oracle.bf_knn(pts, qs, 5, fma=True, threads=8)
    ix = gu.make_index(structure, pts)
    for what in ("tuning call", "tuned call"):
        gu.assert_rows_equal(*gu.run(ix, qs, 5, flags=_lib.QF_AUTOTUNE), *want, what=f"{structure} {what}")
    ix.train_radius_model(gu.to_dev(qs[:512]), 5, steps=20)
    for what in ("tuning call", "tuned call"):
        got = gu.run(ix, qs, 5, flags=_lib.QF_AUTOTUNE | _lib.QF_LEARNED_RADIUS)
        gu.assert_rows_equal(*got, *want, what=f"{structure} learned {what}")
    if structure != "bf":
        for (i, d) in knn.Batch([(ix, gu.to_dev(qs), 5, float("inf"))], autotune=True).run():
            gu.assert_rows_equal(i.cpu().numpy(), d.cpu().numpy(), *want, what=f"{structure} batch")
    ix.close()
