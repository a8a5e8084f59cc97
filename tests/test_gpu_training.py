"""The training step's tiles at their edges: ragged batches (below a tile, one
over, not a multiple of four samples, one over a gradient chunk) against the
numpy reference's gradient, at both widths, and the workspace of ragged
batches."""
from __future__ import annotations

import numpy as np
import pytest

import surrogate_ref as sr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden", [32, 64])
@pytest.mark.parametrize("n", [1, 31, 33, 255, 257, 1874])
def test_gradient_of_ragged_batches(ctx, hidden, n):
    rng = np.random.default_rng(n)
    o = sr.layout(hidden)
    params = rng.normal(0.0, 0.3, o["N_PARAMS"]).astype(np.float32)
    x = rng.uniform(-1.0, 1.0, (n, 5)).astype(np.float32)
    t = rng.normal(0.0, 1.0, (n, 3)).astype(np.float32)
    loss, grad = ctx.surrogate_gradient(params, x, t, hidden)
    ref_loss, ref_grad = sr.loss_and_gradient(params.astype(np.float64), x.astype(np.float64),
                                              t.astype(np.float64))
    # FP32 sums of up to n (hidden) terms: a few n ulp at worst, 1e-5 as for
    # whole batches
    assert loss == pytest.approx(ref_loss, rel=1e-5)
    assert np.abs(grad - ref_grad).max() <= 1e-5 * np.abs(ref_grad).max()


@pytest.mark.parametrize("hidden,batch,steps", [(32, 7, 3), (64, 1001, 5), (64, 257, 4)])
def test_ragged_training_is_reproducible(ctx, kpt, hidden, batch, steps):
    settings = kpt.default_settings(focused=1, closure=kpt.CLOSURE_SURROGATE)
    runs = []
    for _ in range(2):
        net = ctx.train_surrogate(settings, samples=997, steps=steps, batch=batch,
                                  hidden_width=hidden)
        runs.append(net.parameters()[0])
        net.close()
    assert np.isfinite(runs[0]).all() and np.array_equal(runs[0], runs[1])
