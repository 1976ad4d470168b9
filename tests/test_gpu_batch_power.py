"""The step size of a batch's matrices: few large matrices run their power iteration on a
cluster of CTAs, many of them on one CTA each.  The same LP uploaded either way gives the same
iterates; the sums of squares are taken in another order, so the step size may differ by a few
units of 2^-53 and the iterates after 128 iterations by far less than 1e-9."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(1500, 4096, 4), (1501, 4097, 5), (33, 2100, 8), (6000, 9001, 2)])
def test_cluster_and_single_cta_step_size_agree(ctx, lpgen, m, n, k):
    s = lpgen.random_sparse(m=m, n=n, nnz_per_col=k, seed=m).standard()
    assert s.nnz >= 16384

    def solve(copies):
        ctx.batch_upload([(s.m, s.n, s.rowptr, s.colidx, s.vals)] * copies, np.arange(copies, dtype=np.int32),
                         *[np.tile(v, copies) for v in (s.b, s.c, s.lb, s.ub, s.is_eq)])
        _, per, x, y = ctx.batch_solve(precision="fp64", eps=1e-14, max_iterations=128, check_every=64)
        return x[:n], y[:m]

    x1, y1 = solve(1)    # 1 large matrix: a cluster
    x40, y40 = solve(40)  # 40 of them: one CTA each
    assert np.linalg.norm(x1 - x40) <= 1e-9 * np.linalg.norm(x40)
    assert np.linalg.norm(y1 - y40) <= 1e-9 * np.linalg.norm(y40)


@pytest.mark.parametrize("m,n,k,precision", [(2000, 9000, 12, "fp64"), (9000, 24000, 3, "fp32"), (2049, 8160, 5, "fp64")])
def test_cluster_step_size_where_shared_memory_ends(ctx, lpgen, m, n, k, precision):
    """The matrix share of a CTA beyond its shared memory, both vectors beyond it (L2 form; FP32,
    whose iterates also differ by the rounding of the step size), and slices that do not divide by 8."""
    s = lpgen.random_sparse(m=m, n=n, nnz_per_col=k, seed=m).standard()

    def solve(copies):
        ctx.batch_upload([(s.m, s.n, s.rowptr, s.colidx, s.vals)] * copies, np.arange(copies, dtype=np.int32),
                         *[np.tile(v, copies) for v in (s.b, s.c, s.lb, s.ub, s.is_eq)])
        _, per, x, y = ctx.batch_solve(precision=precision, eps=1e-14, max_iterations=128, check_every=64)
        return x[:n], y[:m]

    x1, y1 = solve(1)
    x40, y40 = solve(40)
    tol = 1e-9 if precision == "fp64" else 2e-5
    assert np.linalg.norm(x1 - x40) <= tol * np.linalg.norm(x40)
    assert np.linalg.norm(y1 - y40) <= tol * np.linalg.norm(y40)
