"""Autotuned plans of learned-radius queries belong to the radius model they were tuned with."""

import ctypes

import numpy as np
import pytest

import oracle
from cudaexactknn_gb300 import workloads as W

pytestmark = pytest.mark.gpu
gu = pytest.importorskip("gpu_util")


def _plan(ix, k, learned):
    """The tuned plan's options, or None where there is none yet."""
    from cudaexactknn_gb300 import _lib
    o, ms = _lib.QueryOpts(), ctypes.c_float()
    st = _lib.load().knn_tuned_plan(ix.handle, k, learned, ctypes.byref(o), ctypes.byref(ms))
    return o if st == 0 else None


def _learned_index(structure, dims):
    rng = np.random.default_rng(dims)
    pts, centres = W.mixture(rng, 30000, dims, 16, 0.01)
    qs, _ = W.mixture(rng, 4000, dims, 16, 0.01, centres)
    ix = gu.make_index(structure, pts, 1)
    ix.train_radius_model(gu.to_dev(qs[:1000]), 10, steps=50)
    return ix, qs, oracle.bf_knn(pts, qs, 10, fma=True, threads=8)


@pytest.mark.parametrize("structure", ["kd", "ball", "bf"])
def test_a_new_model_is_tuned_anew(structure):
    from cudaexactknn_gb300 import _lib
    ix, qs, want = _learned_index(structure, 3)
    learned = _lib.QF_AUTOTUNE | _lib.QF_LEARNED_RADIUS

    def tune():
        gu.assert_rows_equal(*gu.run(ix, qs, 10, flags=learned), *want)
        gu.assert_rows_equal(*gu.run(ix, qs, 10, flags=_lib.QF_AUTOTUNE), *want)
        assert _plan(ix, 10, 1) is not None and _plan(ix, 10, 0) is not None
    tune()
    ix.train_radius_model(gu.to_dev(qs[:1000]), 10, steps=60)
    assert _plan(ix, 10, 1) is None and _plan(ix, 10, 0) is not None
    tune()
    ix.import_radius_model(ix.export_radius_model(), 10)
    assert _plan(ix, 10, 1) is None and _plan(ix, 10, 0) is not None
    tune()
    ix.close()


@pytest.mark.parametrize("structure", ["kd", "ball", "bf"])
def test_a_plan_says_whether_it_uses_the_seeds(structure):
    """With seeds that hold nothing, a plan that uses them counts every query as short; one that does not, none."""
    from cudaexactknn_gb300 import _lib, knn
    ix, qs, want = _learned_index(structure, 3)
    params = ix.export_radius_model()
    params[-1] -= 30
    ix.import_radius_model(params, 10)
    learned = _lib.QF_AUTOTUNE | _lib.QF_LEARNED_RADIUS
    gu.assert_rows_equal(*gu.run(ix, qs, 10, flags=learned), *want)
    gu.assert_rows_equal(*gu.run(ix, qs, 10, flags=_lib.QF_AUTOTUNE), *want)
    short = ix.stats(knn.Query(gu.to_dev(qs), len(qs), float("inf")), 10, flags=learned).fallback_queries
    assert bool(_plan(ix, 10, 1).flags & _lib.QF_LEARNED_RADIUS) == (short > len(qs) // 2)
    assert not _plan(ix, 10, 0).flags & _lib.QF_LEARNED_RADIUS
    ix.close()
