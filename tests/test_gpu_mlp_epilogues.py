"""The loss epilogue of the output layer, the column sums and the Adam kernel at the edges of
their tiles, against the FP64 oracle (gradients to BF16 rounding, as for whole batches) and
against Adam in FP64 from the same gradients."""
from __future__ import annotations

import numpy as np
import pytest

import mlp_oracle as mo

pytestmark = pytest.mark.gpu

EDGES = [(8, 8, 1, 1), (64, 72, 127, 7), (64, 128, 128, 64), (72, 136, 129, 65), (64, 128, 257, 129), (256, 256, 1001, 200)]


def segments(i, h, o):
    return [h * i, h, h * h, h, o * h, o]


@pytest.mark.parametrize("i,h,o,n", EDGES)
def test_gradient_at_tile_edges(ctx, i, h, o, n):
    rng = np.random.default_rng(i + h + o + n)
    ctx.mlp_create(i, h, o, seed=3)
    flat = (rng.standard_normal(ctx.mlp_param_count()) * 0.1).astype(np.float32)
    ctx.mlp_set_params(flat)
    X = rng.standard_normal((n, i)).astype(np.float32)
    T = rng.standard_normal((n, o)).astype(np.float32)
    loss, g = ctx.mlp_gradient(X, T)
    loss_ref, grads = mo.loss_and_grad(flat, X.astype(np.float64), T.astype(np.float64), i, h, o)
    assert abs(loss - loss_ref) <= 1e-3 * loss_ref + 1e-12
    s = 0
    for name, gr in zip(("W1", "b1", "W2", "b2", "W3", "b3"), grads):
        gg = g[s:s + gr.size].reshape(gr.shape)
        s += gr.size
        rel = np.linalg.norm(gg - gr) / max(np.linalg.norm(gr), 1e-30)
        assert rel <= 2e-2, (name, rel)


@pytest.mark.parametrize("i,h,o,n", EDGES)
def test_one_adam_step_at_tile_edges(ctx, i, h, o, n):
    """The first step from the gradient the library itself reports: m = 0.1 g, v = 0.001 g^2,
    w -= lr (m / 0.1) / (sqrt(v / 0.001) + 1e-8); 1 - 0.999 in FP32 is 2^-24 / 0.001 = 6e-5 off,
    half of that in the square root, so the update is within 1e-4 of lr."""
    rng = np.random.default_rng(i * h + o + n)
    ctx.mlp_create(i, h, o, seed=3)
    flat = (rng.standard_normal(ctx.mlp_param_count()) * 0.1).astype(np.float32)
    ctx.mlp_set_params(flat)
    X = rng.standard_normal((n, i)).astype(np.float32)
    T = rng.standard_normal((n, o)).astype(np.float32)
    _, g = ctx.mlp_gradient(X, T)
    lr = 1e-3
    ctx.mlp_train_epoch(X, T, batch=n, lr=lr)
    g = g.astype(np.float64)
    want = flat - lr * g / (np.abs(g) + 1e-8)
    assert np.abs(ctx.mlp_get_params() - want).max() <= 1e-4 * lr + 1e-7
