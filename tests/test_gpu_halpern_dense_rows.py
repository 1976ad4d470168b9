"""Rows and columns far longer than the others: the check copies of the single-LP engine leave them out, and
whole CTAs sum them over the CSR arrays in the power iteration, the KKT checks and the certificates."""
from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spl

import pdlp_oracle

pytestmark = pytest.mark.gpu


def dense_lp(lpgen, m, n, k, rows, cols, seed=0):
    """About k entries per column, row 7 i with rows[i] entries, column 5 j with cols[j]; feasible, boxed."""
    rng = np.random.default_rng(seed)
    r, c = [rng.integers(0, m, n * k)], [np.repeat(np.arange(n), k)]
    keep = ~np.isin(r[0], 7 * np.arange(len(rows))) & ~np.isin(c[0], 5 * np.arange(len(cols)))
    r[0], c[0] = r[0][keep], c[0][keep]
    for i, cnt in enumerate(rows):
        r.append(np.full(cnt, i * 7))
        c.append(len(cols) * 5 + rng.choice(n - len(cols) * 5, cnt, replace=False))
    for j, cnt in enumerate(cols):
        r.append(len(rows) * 7 + rng.choice(m - len(rows) * 7, cnt, replace=False))
        c.append(np.full(cnt, j * 5))
    key = np.unique(np.concatenate(r).astype(np.int64) * n + np.concatenate(c))
    r, c = key // n, (key % n).astype(np.int32)
    v = rng.uniform(0.1, 10.0, len(c)) * rng.choice([-1.0, 1.0], len(c))
    eq = np.arange(m) % 2 == 0
    b = np.bincount(r, weights=v * rng.random(n)[c], minlength=m) + np.where(eq, 0.0, rng.random(m))
    ptr = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=m))]).astype(np.int32)
    return lpgen.StdLP(m, n, ptr, c, v, b, rng.uniform(-1.0, 1.0, n), np.zeros(n), np.full(n, 10.0), eq.astype(np.uint8))


CASES = [
    (800, 3000, 3, [256, 257, 3000], []),          # one entry on either side of the limit, and a full row
    (3000, 900, 3, [], [256, 257, 2900]),           # the same for columns
    (2000, 3000, 3, [2900] * 9, [1900] * 3),        # both, more long rows than fit one slice of 8
    (80001, 30000, 8, [20000, 400], [70000]),       # check copies of 16-row slices
    (152000, 160000, 4, [100000], [150000, 1000]),  # of 32-row slices
]


@pytest.mark.parametrize("m,n,k,rows,cols", CASES)
def test_step_size_and_residuals_with_long_rows(ctx, lpgen, m, n, k, rows, cols):
    lp = dense_lp(lpgen, m, n, k, rows, cols)
    dr, dc = pdlp_oracle.ruiz_pc_scaling(lp)
    A = sp.diags(dr) @ sp.csr_matrix((lp.vals, lp.colidx, lp.rowptr), (m, n)) @ sp.diags(dc)
    s2, s1 = np.sort(spl.svds(A, k=2, return_singular_vectors=False, tol=1e-10, random_state=0))
    # The power iteration stops at a relative change of 1e-7 a step; with errors shrinking by
    # rho = (s2 / s1)^2 a step, at most 1e-7 rho / (1 - rho) of sigma^2 are then missing, or rho^1024 at its cap of 512.
    rho = (s2 / s1) ** 2
    missing = max(1e-7 * rho / (1 - rho), rho ** 1024)
    assert missing < 0.05
    ctx.upload(lp)
    for precision in ("fp64", "fp32"):
        r, x, y = ctx.solve(engine="halpern", precision=precision, eps=0.0, max_iterations=128, check_every=64)
        assert 1 - 1e-9 <= r["step_size"] * s1 / 0.998 <= 1 + missing + 1e-9
        kkt = pdlp_oracle.kkt(lp, x, y)
        # sums of up to 150,000 terms in FP64, in another order
        for field, key in (("rel_primal_residual", "rel_primal"), ("rel_dual_residual", "rel_dual"), ("rel_gap", "rel_gap")):
            assert abs(r[field] - kkt[key]) <= 1e-9 * (1 + kkt[key]), (precision, key, r[field], kkt[key])


@pytest.mark.parametrize("kind", ["infeasible", "unbounded"])
def test_certificates_with_a_long_row_and_column(ctx, lpgen, kind):
    lp = dense_lp(lpgen, 1500, 3000, 3, [2900], [1400], seed=3)
    row = slice(lp.rowptr[0], lp.rowptr[1])
    if kind == "infeasible":  # row 0: a sum of boxed columns that is never so large
        lp.is_eq[0] = 0
        lp.vals[row] = -1.0
        lp.b[0] = -(10.0 * (row.stop - row.start) + 1000.0)
    else:  # column 0: it improves the objective and only relaxes its rows
        lp.is_eq[:] = 0
        lp.vals[lp.colidx == 0] = -np.abs(lp.vals[lp.colidx == 0])
        lp.c[0], lp.ub[0] = -1.0, np.inf
    ctx.upload(lp)
    for precision in ("fp64", "fp32"):
        r, _, _ = ctx.solve(engine="halpern", precision=precision, eps=1e-8, eps_infeasible=1e-6, max_iterations=20000)
        assert r["status"] == ("INFEASIBLE_DETECTED" if kind == "infeasible" else "UNBOUNDED_DETECTED")
