"""Long rows and columns of the reference engine are summed by whole warps, in entry order all the same: the
iterates are the oracle's bit for bit in every form."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def lp_with(lpgen, m, n, k, rows, cols, seed):
    """About k entries a column; row 7 i has exactly rows[i] entries, column 5 j exactly cols[j]."""
    rng = np.random.default_rng(seed)
    r, c = rng.integers(0, m, n * k), np.repeat(np.arange(n), k)
    keep = ~np.isin(r, 7 * np.arange(len(rows))) & ~np.isin(c, 5 * np.arange(len(cols)))
    r, c = [r[keep]], [c[keep]]
    others = np.setdiff1d(np.arange(n), 5 * np.arange(len(cols)))
    for i, cnt in enumerate(rows):
        r.append(np.full(cnt, 7 * i)), c.append(rng.choice(others, cnt, replace=False))
    others = np.setdiff1d(np.arange(m), 7 * np.arange(len(rows)))
    for j, cnt in enumerate(cols):
        r.append(rng.choice(others, cnt, replace=False)), c.append(np.full(cnt, 5 * j))
    key = np.unique(np.concatenate(r).astype(np.int64) * n + np.concatenate(c))
    r, c = key // n, (key % n).astype(np.int32)
    v = rng.uniform(0.1, 10.0, len(c)) * rng.choice([-1.0, 1.0], len(c))
    eq = np.arange(m) % 2 == 0
    b = np.bincount(r, weights=v * rng.random(n)[c], minlength=m) + np.where(eq, 0.0, rng.random(m))
    ptr = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=m))]).astype(np.int32)
    return lpgen.StdLP(m, n, ptr, c, v, b, rng.uniform(-1.0, 1.0, n), np.zeros(n), np.full(n, 10.0), eq.astype(np.uint8))


@pytest.mark.parametrize("m,n,k,rows,cols", [
    (60, 300, 3, [128, 129, 160, 161, 299], []), (300, 200, 3, [], [128, 129, 255, 256, 257]),  # one CTA
    (33, 2000, 1, [2000], []),                                    # a slice of nothing but one long row
    (1500, 4500, 6, [1400, 129], [1400]),                         # a cluster
    (700, 3000, 2, [130] * 95, []), (2000, 900, 2, [], [150] * 120),  # many rows of a usual length
    (2000, 900, 2, [400] * 60, [300] * 20), (2500, 7000, 6, [1200] * 3, [900] * 5),
    (3001, 9001, 6, [9000, 300], [2900]), (20011, 30013, 6, [9000] * 2, [130, 20000]),  # two kernels
    (3500, 1000, 1, [900] + [120 if i % 5 == 0 else 1 for i in range(499)], []),  # ... over the CSR arrays
])
def test_long_rows_match_the_oracle(ctx, lpgen, oracle, m, n, k, rows, cols):
    s = lp_with(lpgen, m, n, k, rows, cols, seed=m + n)
    ctx.upload(s)
    for iterations, cf in ((130, 100), (43, 7)):
        res, x, y = ctx.solve(engine="reference", max_iterations=iterations, check_frequency=cf)
        o = oracle.ref_pdhg(s, max_iterations=iterations, check_frequency=cf)
        assert res["iterations"] == o["iterations"] and res["used_average"] == o["used_average"]
        assert np.array_equal(x, o["x_final"]) and np.array_equal(y, o["y_last"])

