"""The radius model's forward, backward and update kernels where a batch or a layer ends: samples per
forward block (8), per gradient tile (64) and step (8), input columns per warp.

Tolerance, derived: a gradient is a sum of at most 1,030 float products of values that carry the rounding of
three chains of at most 192 terms and of the projections' phase (2 pi a with |a| up to about 40: 2.4e-5
absolute in sin and cos); 1,400 units of 2^-24 and that phase error on terms up to the layer's scale bound the
error by 1.2e-4 of the largest gradient, relative 2e-3 where a ReLU's sign agrees (the model's own test's)."""

import numpy as np
import pytest

import radius_model_ref as ref

pytestmark = pytest.mark.gpu
gu = pytest.importorskip("gpu_util")


def _params(d, rng):
    n = 64 * (d + 64) + 64 + 64 * 64 + 64 + 64 + 1
    p = np.zeros(n + 32 * d + 2 * d + 1, np.float32)
    p[:n] = rng.standard_normal(n).astype(np.float32) * 0.2
    p[n:n + 32 * d] = rng.standard_normal(32 * d) * 4.0 / np.sqrt(d)
    p[n + 33 * d:n + 34 * d] = 1.0
    return p


@pytest.mark.parametrize("batch", [1, 7, 9, 63, 64, 65, 129, 1030])
@pytest.mark.parametrize("d", [1, 3, 32, 33, 128])
def test_batch_and_layer_ends(d, batch):
    from cudaexactknn_gb300 import knn
    rng = np.random.default_rng(1000 * d + batch)
    p = _params(d, rng)
    x = rng.random((batch, d)).astype(np.float32)
    t = rng.standard_normal(batch).astype(np.float32)
    loss, grad = knn.radius_model_gradients(p, d, x, t)
    want_loss, want = ref.loss_and_grad(p, d, x, t)
    assert abs(loss - want_loss) <= 1e-4 * max(1.0, abs(want_loss))
    np.testing.assert_allclose(grad, want, rtol=2e-3, atol=1.2e-4 * np.abs(want).max())


def test_training_repeats_and_uses_every_batch():
    """The same samples train the same model, bit for bit, also with a batch that is no multiple of a tile."""
    from cudaexactknn_gb300 import workloads as W
    rng = np.random.default_rng(2)
    pts = W.uniform(rng, 3000, 3)
    samples = gu.to_dev(W.uniform(rng, 700, 3))
    got = []
    for _ in range(2):
        ix = gu.make_index("kd", pts)
        rep = ix.train_radius_model(samples, 5, steps=40, batch=333)
        got.append(ix.export_radius_model())
        assert rep.samples == 700 and rep.steps == 40
        ix.close()
    np.testing.assert_array_equal(got[0].view(np.uint32), got[1].view(np.uint32))
