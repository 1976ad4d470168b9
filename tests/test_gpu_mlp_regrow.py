"""A captured training epoch and calls between two trainings that move its buffers."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,rows", [(64, (104, 4096)), (64, (97, 200, 1000)), (256, (136, 2048))])
def test_training_goes_on_after_larger_requests(b2p, lpgen, hidden, rows):
    """Training, inference and gradients of more rows, training: the same parameters bit for bit as with
    buffers that were large enough from the start."""
    s = lpgen.random_sparse(m=40, n=90, nnz_per_col=3, seed=1).standard()
    count, out = 300, s.n + s.m + 1
    rng = np.random.default_rng(2)
    costs, feats = rng.uniform(-1.0, 1.0, count * s.n), rng.uniform(0.5, 1.5, (count, 16)).astype(np.float32)
    big = rng.standard_normal((max(rows), 16)).astype(np.float32)

    def train(large_first):
        c = b2p.Context(0)
        try:
            c.batch_upload([(s.m, s.n, s.rowptr, s.colidx, s.vals)], np.zeros(count, np.int32), np.tile(s.b, count),
                           costs, np.tile(s.lb, count), np.tile(s.ub, count), np.tile(s.is_eq, count))
            c.batch_solve(precision="fp32", max_iterations=64, check_every=64, outputs=False)
            c.mlp_create(16, hidden, out, seed=5)
            c.mlp_dataset_from_batch(feats)
            if large_first:
                c.mlp_gradient(big, np.zeros((len(big), out), np.float32))
            for r in rows:
                c.mlp_train(2, batch=96, seed=3)
                c.mlp_infer(big[:r])
                c.mlp_gradient(big[:r], np.zeros((r, out), np.float32))
            c.mlp_train(2, batch=96, seed=4)
            return c.mlp_get_params()
        finally:
            c.close()

    a, b = train(False), train(True)
    assert np.all(np.isfinite(a)) and np.array_equal(a, b)
