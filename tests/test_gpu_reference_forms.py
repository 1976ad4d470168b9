"""The forms of the reference engine -- one CTA, a cluster with the matrix in shared memory or
outside it, two kernels per iteration over sliced or CSR copies -- are the oracle's iteration
bit for bit, at sizes around a slice of 32, at the borders between the forms, with rows that
make a sliced copy too long, and when the iterates diverge."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def dense_row(lp, rng, entries):
    """The LP with row 0 holding `entries` entries."""
    rows = [(lp.colidx[lp.rowptr[i]:lp.rowptr[i + 1]], lp.vals[lp.rowptr[i]:lp.rowptr[i + 1]]) for i in range(lp.m)]
    rows[0] = (np.arange(entries, dtype=np.int32), rng.uniform(0.1, 1.0, entries))
    lp.rowptr = np.concatenate([[0], np.cumsum([len(r[0]) for r in rows])]).astype(np.int32)
    lp.colidx = np.concatenate([r[0] for r in rows])
    lp.vals = np.concatenate([r[1] for r in rows])
    return lp


@pytest.mark.parametrize("m,n,k,dense,iterations,cf", [
    (1, 3, 1, 0, 250, 100), (31, 33, 3, 0, 137, 7), (32, 64, 4, 0, 201, 100), (33, 65, 5, 0, 199, 100),
    (64, 200, 4, 0, 1, 100), (257, 900, 5, 0, 150, 50),          # one CTA, then a cluster
    (300, 1001, 5, 0, 300, 100), (1500, 4500, 6, 0, 130, 100),    # a cluster
    (700, 16000, 3, 0, 120, 100), (2047, 7000, 7, 0, 120, 100),   # at the borders of the forms
    (3001, 9001, 6, 0, 150, 100), (9001, 20003, 3, 0, 110, 100),  # two kernels per iteration
    (40, 3000, 1, 3000, 120, 100), (3000, 9000, 1, 9000, 120, 100),  # padding too long: CSR
])
def test_reference_forms_match_oracle(ctx, lpgen, oracle, m, n, k, dense, iterations, cf):
    s = lpgen.random_sparse(m=m, n=n, nnz_per_col=k, seed=m + n).standard()
    if dense:
        s = dense_row(s, np.random.default_rng(m), dense)
    ctx.upload(s)
    res, x, y = ctx.solve(engine="reference", max_iterations=iterations, check_frequency=cf)
    o = oracle.ref_pdhg(s, max_iterations=iterations, check_frequency=cf)
    assert res["iterations"] == o["iterations"] and res["used_average"] == o["used_average"]
    assert np.array_equal(x, o["x_final"]) and np.array_equal(y, o["y_last"])


@pytest.mark.parametrize("m,n", [(60, 200), (300, 1000), (3001, 9001)])
def test_reference_forms_diverge_like_the_oracle(ctx, lpgen, oracle, m, n):
    """Steps beyond the stable ones: the iterates grow past 1e15 and the failure is found at the
    same check."""
    s = lpgen.random_sparse(m=m, n=n, nnz_per_col=5, seed=5).standard()
    s.ub = np.full(n, np.inf)
    ctx.upload(s)
    args = dict(adaptive_step_size=0, primal_step_size=0.5, dual_step_size=0.5)
    res, _, _ = ctx.solve(engine="reference", max_iterations=1000, **args)
    o = oracle.ref_pdhg(s, max_iterations=1000, adaptive=False, primal_step=0.5, dual_step=0.5)
    assert res["iterations"] == o["iterations"]
    assert res["status"] == o["status"]


@pytest.mark.parametrize("m,n,k", [(2000, 100, 60), (3000, 33, 100), (180, 600, 5), (205, 615, 5)])
def test_cluster_ctas_without_columns_match_oracle(ctx, lpgen, oracle, m, n, k):
    """A cluster with fewer column slices than CTAs (the empty ones post a token), and the two sides of
    one CTA / cluster (3,072 entries): bit for bit over two check intervals and a remainder."""
    s = lpgen.random_sparse(m=m, n=n, nnz_per_col=k, seed=m + n).standard()
    ctx.upload(s)
    res, x, y = ctx.solve(engine="reference", max_iterations=230)
    o = oracle.ref_pdhg(s, max_iterations=230)
    assert res["iterations"] == o["iterations"] and res["status"] == o["status"]
    assert np.array_equal(x, o["x_final"]) and np.array_equal(y, o["y_last"])
