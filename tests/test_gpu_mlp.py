"""The predictor's training kernel at the sizes where its tiles (32 samples),
staged chunks (64) and clusters (16 tiles) end: the full-batch gradient
against the numpy reference (rtol 2e-4 with the gradient's scale as atol, as
in test_gpu_learned), and one optimiser step -- whose moments start at zero,
so that every parameter moves by lr g / (|g| + 1e-8) against its gradient."""
from __future__ import annotations

import numpy as np
import pytest

import mlp_reference as ref

pytestmark = pytest.mark.gpu


def _data(n):
    rng = np.random.default_rng(n)
    x = rng.normal(0, 1, (n, 10)).astype(np.float32)
    y = (0.3 * x[:, 0] - 0.2 * np.tanh(x[:, 1]) + 0.1 * x[:, 2] * x[:, 3]).astype(np.float32)
    return x, y


@pytest.mark.parametrize("n", [2, 31, 32, 33, 64, 65, 511, 512, 513, 1100])
def test_gradient_and_step_at_tile_edges(engine_lib, n):
    from periodsearch_gb300 import learned

    x, y = _data(n)
    P = learned.init_weights(x, y, seed=1)
    loss, g = learned.grad(P, x, y)
    loss_r, g_r = ref.loss_grad(P, x, y)
    assert abs(loss - loss_r) <= 1e-4 * abs(loss_r)
    scale = np.abs(g_r).max()
    np.testing.assert_allclose(g, g_r, rtol=2e-4, atol=2e-5 * scale)
    lr = 1e-3
    W, hist = learned.train(x, y, epochs=1, batch=n, lr=lr, weights=P)
    assert abs(hist[0] - loss) <= 1e-5 * abs(loss)
    clear = np.abs(g_r) > 1e-3 * scale   # far from zero: the sign is certain
    np.testing.assert_allclose((W - P)[clear], -lr * np.sign(g_r[clear]), rtol=1e-2)
    np.testing.assert_array_equal(W[g == 0], P[g == 0])


def test_batches_do_not_depend_on_what_follows(engine_lib):
    """Two epochs of three batches and a remainder that is left out: the
    same weights whether or not more epochs follow."""
    from periodsearch_gb300 import learned

    x, y = _data(100)
    P = learned.init_weights(x, y, seed=2)
    a, ha = learned.train(x, y, epochs=2, batch=33, weights=P, seed=4)
    b, hb = learned.train(x, y, epochs=3, batch=33, weights=P, seed=4)
    np.testing.assert_array_equal(ha, hb[:2])
    assert not np.array_equal(a, b) and np.isfinite(b).all()
