"""The query path's radius prediction (16-bit operands on the tensor cores) at the ends of its operand rows:
coordinates that fill part of a chunk of eight, of a K step of sixteen and of the second 64-wide block; tiles of
128 queries that are full, short and several per block's turn.

The training report's margin and RMSE come from these predictions.  The oracle restates them in float64 on
operands rounded to 16 bits.  Tolerance, derived: what is left are operands that round to the other neighbour
(a difference of 2^-10 relative at most, each with its own sign) and single-precision sums, which are smaller;
six standard deviations of the independent roundings, carried through both layers, bound a prediction's error,
the largest over the samples bounds the quantile's and the RMSE's, and the logarithm's own 1e-5 is added."""

import numpy as np
import pytest

import radius_model_ref as ref

pytestmark = pytest.mark.gpu
gu = pytest.importorskip("gpu_util")


def _half(v):
    return np.asarray(v, np.float64).astype(np.float16).astype(np.float64)


def _predict(params, d, x):
    m = ref.split(params, d)
    e, w1, w2 = _half(ref.features(m, x)), _half(m["W1"]), _half(m["W2"])
    h1 = _half(np.maximum(e @ w1.T + m["b1"], 0))
    h2 = np.maximum(h1 @ w2.T + m["b2"], 0)
    u = 2.0 ** -10
    var1 = (u * e) ** 2 @ (w1 ** 2).T + (u * h1) ** 2
    var2 = var1 @ (w2 ** 2).T
    return h2 @ m["w3"] + m["b3"], 6.0 * np.sqrt(var2 @ (m["w3"] ** 2))


@pytest.mark.parametrize("d,count", [(1, 127), (3, 128), (4, 300), (5, 129), (8, 300), (9, 300), (16, 300), (17, 300),
                                     (32, 300), (33, 300), (63, 300), (64, 300), (3, 150000)])
def test_margin_and_rmse(d, count):
    from cudaexactknn_gb300 import workloads as W
    rng = np.random.default_rng(10 * d + 1)
    pts, centres = W.mixture(rng, 4000, d, 8, 0.05)
    samples, _ = W.mixture(rng, count, d, 8, 0.05, centres)
    ix = gu.make_index("bf", pts)
    rep = ix.train_radius_model(gu.to_dev(samples), 3, steps=60, coverage=0.5)
    _, dist = gu.run(ix, samples, 3)
    pred, tol = _predict(ix.export_radius_model(), d, samples)
    resid = np.log(np.maximum(np.asarray(dist, np.float64)[:, -1], 1e-30)) - pred
    bound = float(tol.max()) + 1e-5
    order = np.sort(resid)
    want = order[min(count - 1, int(np.ceil(0.5 * count)))] + 1e-3
    assert abs(rep.margin - want) <= bound
    assert abs(rep.rmse - np.sqrt(np.mean(resid ** 2))) <= bound
    ix.close()
