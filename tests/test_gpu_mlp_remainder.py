"""Training epochs whose last batch is shorter than the others.  Fewer rows can want more split-K
workspace than a full batch, and the epoch is captured as a graph, in which nothing may grow."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def train(b2p, lpgen, count, batch, grow_first):
    """Parameters and loss after two epochs on the labels of a batch of planning-sized LPs (out = 10,001)."""
    s = lpgen.random_sparse(m=2000, n=8000, nnz_per_col=3, seed=1).standard()
    rng = np.random.default_rng(2)
    c = b2p.Context(0)
    try:
        c.batch_upload([(s.m, s.n, s.rowptr, s.colidx, s.vals)], np.zeros(count, np.int32), np.tile(s.b, count),
                       rng.uniform(-1.0, 1.0, count * s.n), np.tile(s.lb, count), np.tile(s.ub, count),
                       np.tile(s.is_eq, count))
        c.batch_solve(precision="fp32", max_iterations=64, check_every=64, outputs=False)
        c.mlp_create(256, 1024, s.n + s.m + 1, seed=5)
        c.mlp_dataset_from_batch(rng.uniform(0.5, 1.5, (count, 256)).astype(np.float32))
        if grow_first:  # every row count of the epoch, outside the training call
            for rows in {min(batch, count), count % batch or batch}:
                c.mlp_gradient(np.zeros((rows, 256), np.float32), np.zeros((rows, s.n + s.m + 1), np.float32))
        return c.mlp_train(2, batch=batch, seed=3), c.mlp_get_params()
    finally:
        c.close()


@pytest.mark.parametrize("count,batch", [
    (640, 512),   # remainder 128: 2,359,296 floats against 2,097,152 of a full batch
    (1250, 1024),  # 226, padded to 232
    (500, 512),   # one short batch
])
def test_training_with_a_short_last_batch(b2p, lpgen, count, batch):
    """The same parameters bit for bit as with the workspaces grown before the call."""
    loss, params = train(b2p, lpgen, count, batch, False)
    loss2, params2 = train(b2p, lpgen, count, batch, True)
    assert np.isfinite(loss) and np.all(np.isfinite(params))
    assert np.array_equal(params, params2) and abs(loss - loss2) <= 1e-6 * abs(loss2)
