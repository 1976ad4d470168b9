"""Small LPs iterate between checks in one launch (one CTA, or a cluster): the same iteration as
the two kernels per iteration that ``lanes_per_row`` asks for, up to the order of the sums."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# the smallest; slices that are full, one over and one short; both sides of one CTA / cluster (256
# columns) and of one CTA's limit (8,192 entries); a cluster with fewer row slices than CTAs; rows past
# the longest (two kernels); the largest that fit, FP32 and FP64, and one that fits neither
SHAPES = [(1, 2, 1), (31, 32, 2), (33, 65, 3), (300, 255, 32), (300, 255, 33), (300, 256, 5), (300, 1000, 5),
          (97, 1500, 5), (60, 1000, 8), (40, 4200, 3), (1500, 5000, 6), (2000, 8000, 6), (3001, 12190, 6)]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_one_launch_form_matches_two_kernels(ctx, lpgen, m, n, k, precision):
    """256 iterations, checks every 64 and every 7 (restart checks, and with FP32 the re-centring,
    included).  The operator is non-expansive, so the points differ by the rounding of about 256
    iterations of k-entry sums: 256 * 20 * 2^-53 (FP64), 256 * 20 * 2^-24 of a correction (FP32)."""
    lp = lpgen.random_sparse(m, n, k, seed=m + n).standard()
    tol = 1e-10 if precision == "fp64" else 4e-4
    for every in (64, 7):
        ctx.upload(lp)
        kw = dict(engine="halpern", precision=precision, eps=0.0, max_iterations=256, check_every=every)
        ra, xa, ya = ctx.solve(**kw)
        rb, xb, yb = ctx.solve(lanes_per_row=-1, **kw)
        assert ra["iterations"] == rb["iterations"] and ra["restarts"] == rb["restarts"]
        assert np.linalg.norm(xa - xb) <= tol * (1 + np.linalg.norm(xb))
        assert np.linalg.norm(ya - yb) <= tol * (1 + np.linalg.norm(yb))
        assert abs(ra["rel_kkt"] - rb["rel_kkt"]) <= 10 * tol * (1 + rb["rel_kkt"])


def test_kernel_timing_after_one_launch_solve(ctx, lpgen):
    """b2p_kernel_timing times the two kernels of an LP whose solve used neither."""
    ctx.upload(lpgen.random_sparse(300, 1000, 5, seed=1).standard())
    ctx.solve(engine="halpern", precision="fp64", eps=0.0, max_iterations=128)
    t = ctx.kernel_timing(reps=3, precision="fp64")
    assert all(v > 0 for v in (t.values() if isinstance(t, dict) else t))
