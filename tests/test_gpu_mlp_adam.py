"""Several Adam steps on different batches, whose update depends on the gradients' size: the split partial
sums that Adam reads are those that the gradient call adds up."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("i,h,o,n", [
    (64, 128, 40, 48),       # no GEMM is split
    (256, 256, 136, 1024),   # the gradients of W1 and W2 in four parts each
    (64, 64, 72, 1000),      # ... with a remainder
    (256, 1024, 1001, 520),  # W1 alone
])
def test_adam_steps_match_fp64_adam_of_the_gradients(ctx, i, h, o, n):
    """Each step from the weights before it.  m and v are within a few 2^-24 of their largest terms a step,
    1 - 0.999^t in FP32 within 2^-24 / (0.001 t) = 6e-5 / t, half of that in the square root; an update is at
    most 0.1 / sqrt(0.001) = 3.2 times lr.  So 2e-4 lr, and the rounding of a weight of up to 1."""
    rng = np.random.default_rng(i + h + o + n)
    ctx.mlp_create(i, h, o, seed=3)
    w = (rng.standard_normal(ctx.mlp_param_count()) * 0.1).astype(np.float32)
    ctx.mlp_set_params(w)
    m, v = np.zeros(w.size), np.zeros(w.size)
    lr = 1e-2
    for t in range(1, 5):
        X = (rng.standard_normal((n, i)) * t).astype(np.float32)
        T = (rng.standard_normal((n, o)) * 3.0 / t).astype(np.float32)
        _, g = ctx.mlp_gradient(X, T)
        g = g.astype(np.float64)
        ctx.mlp_train_epoch(X, T, batch=n, lr=lr)
        m = 0.9 * m + 0.1 * g
        v = 0.999 * v + 0.001 * g * g
        want = w - lr * (m / (1 - 0.9**t)) / (np.sqrt(v / (1 - 0.999**t)) + 1e-8)
        w = ctx.mlp_get_params()
        assert np.abs(w - want).max() <= 2e-4 * lr + 2.0**-23
        # the state the library holds differs from this one by roundings only; go on from its own weights
