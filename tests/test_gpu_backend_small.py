"""The small forms of the GpuBackend primitives -- one packed copy each way, A^T y in one CTA
without a transpose -- are the host loops bit for bit, at the borders to the general forms, and
refuse what the general forms refuse."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (3, 40, 2), (33, 31, 6), (300, 1000, 5), (700, 3072, 4), (700, 3073, 4),
                                   (1024, 8192, 1), (1025, 8192, 1), (64, 8193, 1), (20000, 60000, 1), (2, 12000, 1)])
def test_spmv_forms_match_the_host_loops(ctx, lpgen, oracle, m, n, k):
    s = lpgen.random_sparse(m=m, n=n, nnz_per_col=k, seed=m + n).standard()
    rng = np.random.default_rng(n)
    x, y = rng.standard_normal(n), rng.standard_normal(m)
    ax, _ = ctx.spmv(m, n, s.rowptr, s.colidx, s.vals, x)
    aty, t = ctx.spmv(m, n, s.rowptr, s.colidx, s.vals, y, transpose=True)
    assert np.array_equal(ax, oracle.spmv(s, x)) and np.array_equal(aty, oracle.spmv_t(s, y))
    assert t["total_gpu_time_ms"] > 0.0


@pytest.mark.parametrize("m,n", [(300, 1000), (9000, 20000)])
def test_invalid_columns_are_refused(b2p, ctx, lpgen, m, n):
    s = lpgen.random_sparse(m=m, n=n, nnz_per_col=2, seed=1).standard()
    row = int(np.argmax(np.diff(s.rowptr)))
    e = int(s.rowptr[row])
    for value in (-1, n, 2**30, int(s.colidx[e + 1])):
        bad = s.colidx.copy()
        bad[e] = value
        for transpose in (False, True):
            with pytest.raises(b2p.B2PError) as err:
                ctx.spmv(m, n, s.rowptr, bad, s.vals, np.ones(m if transpose else n), transpose=transpose)
            assert err.value.code == b2p.INVALID_ARGUMENT and f"row {row}" in str(err.value)


@pytest.mark.parametrize("n", [1, 1000, 43688, 65533, 300001])
def test_vector_operations_on_both_sides_of_the_packing(ctx, n):
    rng = np.random.default_rng(n)
    a, b = rng.standard_normal(n), rng.standard_normal(n)
    assert np.array_equal(ctx.vector_op("add", a, b), a + b) and np.array_equal(ctx.vector_op("sub", a, b), a - b)
    assert np.array_equal(ctx.vector_op("scale", a, alpha=0.3), 0.3 * a)
    assert np.array_equal(ctx.vector_op("axpy", a, b, alpha=0.3), 0.3 * a + b)
    assert abs(ctx.dot(a, b) - np.dot(a, b)) <= 1e-12 * np.abs(a * b).sum()
    assert abs(ctx.norm2(a) - np.linalg.norm(a)) <= 1e-12 * np.linalg.norm(a)
