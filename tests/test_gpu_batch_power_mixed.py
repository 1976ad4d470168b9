"""Large matrices among many small ones: the power iteration of the large ones is dealt to the clusters by
their place among the large, wherever they lie in the batch."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nmat,stride,big", [(20, 19, 2), (90, 18, 5), (120, 3, 37), (120, 3, 38)])
def test_step_sizes_do_not_depend_on_the_place_in_the_batch(ctx, lpgen, nmat, stride, big):
    """Up to 37 large matrices run on clusters, 38 on one CTA each.  Every copy of an LP gets the same
    iterates as the LP uploaded alone, to the rounding of the step size over 128 iterations."""
    large = lpgen.random_sparse(m=1500, n=4097, nnz_per_col=5, seed=1).standard()
    small = lpgen.random_sparse(m=40, n=90, nnz_per_col=3, seed=2).standard()
    assert large.nnz >= 16384 > small.nnz

    def solve(lps):
        cat = [np.concatenate([getattr(s, f) for s in lps]) for f in ("b", "c", "lb", "ub", "is_eq")]
        ctx.batch_upload([(s.m, s.n, s.rowptr, s.colidx, s.vals) for s in lps], np.arange(len(lps), dtype=np.int32), *cat)
        _, _, x, y = ctx.batch_solve(precision="fp64", eps=1e-14, max_iterations=128, check_every=64)
        return (np.split(x, np.cumsum([s.n for s in lps])[:-1]), np.split(y, np.cumsum([s.m for s in lps])[:-1]))

    want = {id(s): [v[0] for v in solve([s])] for s in (large, small)}
    lps = [large if i % stride == 0 and i // stride < big else small for i in range(nmat)]
    assert sum(s is large for s in lps) == big
    x, y = solve(lps)
    for s, xi, yi in zip(lps, x, y):
        wx, wy = want[id(s)]
        assert np.linalg.norm(xi - wx) <= 1e-9 * np.linalg.norm(wx)
        assert np.linalg.norm(yi - wy) <= 1e-9 * np.linalg.norm(wy)
