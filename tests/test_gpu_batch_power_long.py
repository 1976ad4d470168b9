"""Rows and columns of more than 128 entries in the power iteration of a large batch matrix: on a cluster a
whole warp sums each."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def lp_with(lpgen, m, n, k, rows, cols, seed):
    """About k entries a column, row 7 i with rows[i] entries and column 5 j with cols[j]."""
    rng = np.random.default_rng(seed)
    r, c = [rng.integers(0, m, n * k)], [np.repeat(np.arange(n), k)]
    for i, cnt in enumerate(rows):
        r.append(np.full(cnt, 7 * i)), c.append(rng.choice(n, cnt, replace=False))
    for j, cnt in enumerate(cols):
        r.append(rng.choice(m, cnt, replace=False)), c.append(np.full(cnt, 5 * j))
    key = np.unique(np.concatenate(r).astype(np.int64) * n + np.concatenate(c))
    r, c = key // n, (key % n).astype(np.int32)
    v = rng.uniform(0.1, 10.0, len(c)) * rng.choice([-1.0, 1.0], len(c))
    eq = np.arange(m) % 2 == 0
    b = np.bincount(r, weights=v * rng.random(n)[c], minlength=m) + np.where(eq, 0.0, rng.random(m))
    ptr = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=m))]).astype(np.int32)
    return lpgen.StdLP(m, n, ptr, c, v, b, rng.uniform(-1.0, 1.0, n), np.zeros(n), np.full(n, 10.0), eq.astype(np.uint8))


@pytest.mark.parametrize("m,n,k,rows,cols,precision", [
    (2000, 8000, 3, [8000], [], "fp64"), (1500, 4097, 4, [130] * 40, [1400], "fp64"), (700, 3000, 5, [], [600] * 33, "fp64"),
    (150, 4000, 30, [], [], "fp64"),                          # every row is long
    (9000, 24000, 3, [20000], [8000, 129], "fp32"),            # vectors beyond shared memory
])
def test_cluster_and_single_cta_step_size_agree_with_long_rows(ctx, lpgen, m, n, k, rows, cols, precision):
    """One copy of the matrix runs on a cluster, 40 on one CTA each: the same iterates to the rounding of
    the step size over 128 iterations (FP32: of the iterates, which then start from other values)."""
    s = lp_with(lpgen, m, n, k, rows, cols, seed=m)
    assert s.nnz >= 16384 and np.diff(s.rowptr).max() > 128 or cols

    def solve(copies):
        ctx.batch_upload([(s.m, s.n, s.rowptr, s.colidx, s.vals)] * copies, np.arange(copies, dtype=np.int32),
                         *[np.tile(v, copies) for v in (s.b, s.c, s.lb, s.ub, s.is_eq)])
        _, _, x, y = ctx.batch_solve(precision=precision, eps=1e-14, max_iterations=128, check_every=64)
        return x[:n], y[:m]

    x1, y1 = solve(1)
    x40, y40 = solve(40)
    tol = 1e-9 if precision == "fp64" else 2e-5
    assert np.linalg.norm(x1 - x40) <= tol * np.linalg.norm(x40)
    assert np.linalg.norm(y1 - y40) <= tol * np.linalg.norm(y40)
