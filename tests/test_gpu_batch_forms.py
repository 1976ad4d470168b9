"""The forms of the batched chunk kernel -- one, two or four instances of a shared matrix per
CTA -- against each other (bit for bit) and against the FP64 KKT checker, at the sizes and
options where they take different code: column and row counts around a slice of 32, groups
that are not full, rows longer than the warp-cooperative limit, anchors kept or re-centred
away, a reflection other than 1, instances that finish inside a launch."""
from __future__ import annotations

import numpy as np
import pytest

import pdlp_oracle

pytestmark = pytest.mark.gpu


def family(lpgen, m, n, count, dense, seed):
    """`count` LPs over one matrix (optionally with a row of `dense` entries); their costs differ."""
    rng = np.random.default_rng(seed)
    lp = lpgen.random_sparse(m=m, n=n, nnz_per_col=min(4, m), seed=seed)
    if dense:
        A = np.zeros((m, n))
        for i in range(m):
            A[i, lp.colidx[lp.rowptr[i]:lp.rowptr[i + 1]]] = lp.vals[lp.rowptr[i]:lp.rowptr[i + 1]]
        x0 = rng.random(n)
        A[1, :dense] = rng.uniform(0.1, 1.0, dense)
        lp.rhs[1] = A[1] @ x0 + 50.0  # an inactive <= row stays feasible for the other rows' x0
        r, c = np.nonzero(A)
        lp.rowptr = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=m))]).astype(np.int32)
        lp.colidx, lp.vals = c.astype(np.int32), A[r, c]
    s = lp.standard()
    return s, np.tile(s.b, (count, 1)), rng.uniform(-1.0, 1.0, (count, n))


def solve(b2p, monkeypatch, shape, s, B, Cc, **params):
    monkeypatch.setenv("B2P_BATCH_SHAPE", shape)
    count = len(B)
    c = b2p.Context(0)
    try:
        c.batch_upload([(s.m, s.n, s.rowptr, s.colidx, s.vals)], np.zeros(count, np.int32), B.ravel(), Cc.ravel(),
                       np.tile(s.lb, count), np.tile(s.ub, count), np.tile(s.is_eq, count))
        return c.batch_solve(**params)
    finally:
        c.close()


CASES = [
    # m, n, dense row, count, precision, options
    (31, 96, 0, 301, "fp32", {}),
    (33, 97, 0, 302, "fp32", dict(refinement_rounds=0)),
    (64, 250, 140, 299, "fp32", {}),
    (65, 257, 0, 300, "fp32", dict(reflection=0.5)),
    (33, 97, 0, 301, "fp64", {}),
    (64, 250, 140, 299, "fp64", dict(refinement_rounds=1)),
    (2, 5, 0, 303, "fp32", {}),
]


@pytest.mark.parametrize("m,n,dense,count,precision,options", CASES)
def test_forms_agree(b2p, lpgen, tmp_path, monkeypatch, m, n, dense, count, precision, options):
    monkeypatch.setenv("B2P_AUTOTUNE_CACHE", str(tmp_path / "tune.txt"))
    s, B, Cc = family(lpgen, m, n, count, dense, seed=m + n)
    for params in (dict(eps=1e-13, max_iterations=320, check_every=64),   # every instance runs to the cap
                   dict(eps=1e-4, max_iterations=20000, check_every=64)):  # instances finish at different checks
        out = {}
        for shape in ("256,2,1", "256,1,1", "256,2,2", "256,1,2") + (("256,2,4", "256,1,4") if precision == "fp32" else ()):
            summ, per, x, y = solve(b2p, monkeypatch, shape, s, B, Cc, precision=precision, **params, **options)
            assert int(round(summ["used_average"])) == 10 * int(shape[-1]) + int(shape[4])
            out[shape] = (per, x, y)
        p1, x1, y1 = out["256,2,1"]
        for shape, (p, x, y) in out.items():
            assert np.array_equal(p["status"], p1["status"]), shape
            assert np.array_equal(p["iterations"], p1["iterations"]), shape
            assert np.array_equal(x, x1) and np.array_equal(y, y1), shape
    assert np.all(p1["status"] == 0)
    for i in (0, count // 2, count - 1):  # the answers themselves, by the FP64 checker
        inst = type(s)(s.m, s.n, s.rowptr, s.colidx, s.vals, B[i], Cc[i], s.lb, s.ub, s.is_eq)
        k = pdlp_oracle.kkt(inst, x1[i * n:(i + 1) * n], y1[i * m:(i + 1) * m])
        assert k["rel_kkt"] <= 1.05e-4, (i, k)
