"""B2P_BATCH_SHAPE names the shape that runs, from the first launch of a solve to its last."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", ["128,2,1", "256,1,1", "256,2,2"])
@pytest.mark.parametrize("count", [40, 300])
def test_pinned_shape_does_not_depend_on_the_chunk(b2p, lpgen, tmp_path, monkeypatch, shape, count):
    """The order of every sum is a pinned shape's own, so the answers are the same bit for bit however
    many iterations a launch has (the tuned part of a pinned shape), although instances finish at
    different checks and the batch shrinks at different launches."""
    cache = tmp_path / "tune.txt"
    monkeypatch.setenv("B2P_AUTOTUNE_CACHE", str(cache))
    monkeypatch.setenv("B2P_BATCH_SHAPE", shape)
    s = lpgen.random_sparse(m=65, n=257, nnz_per_col=4, seed=3).standard()
    costs = np.random.default_rng(4).uniform(-1.0, 1.0, (count, s.n))

    def solve():
        c = b2p.Context(0)
        try:
            c.batch_upload([(s.m, s.n, s.rowptr, s.colidx, s.vals)], np.zeros(count, np.int32), np.tile(s.b, count),
                           costs.ravel(), np.tile(s.lb, count), np.tile(s.ub, count), np.tile(s.is_eq, count))
            return c.batch_solve(precision="fp64", eps=1e-6, max_iterations=40000)
        finally:
            c.close()

    solve()
    fields = cache.read_text().split()  # key, CTA size, chunk, ...
    out = []
    for chunk in (256, 4096):
        cache.write_text(" ".join([*fields[:2], str(chunk), *fields[3:]]) + "\n")
        summ, per, x, y = solve()
        assert int(round(summ["step_size"])) == int(shape.split(",")[0]) * 100000 + chunk
        out.append((per["iterations"], x, y))
    assert len(set(out[0][0].tolist())) > 1  # instances finish at different checks
    for a, b in zip(*out):
        assert np.array_equal(a, b)
