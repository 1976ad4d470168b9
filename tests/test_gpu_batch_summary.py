"""The instances per CTA that a batched solve reports are those its first launch ran with."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("learned", [False, True])
def test_summary_names_the_form_that_ran(b2p, lpgen, tmp_path, monkeypatch, learned):
    """A tuned shape of four instances per CTA (written into the cache): a batch of 600 starts with it,
    one of 40 runs one instance per CTA from the first launch on."""
    cache = tmp_path / "tune.txt"
    monkeypatch.setenv("B2P_AUTOTUNE_CACHE", str(cache))
    monkeypatch.delenv("B2P_BATCH_SHAPE", raising=False)
    s = lpgen.random_sparse(m=64, n=250, nnz_per_col=4, seed=3).standard()
    rng = np.random.default_rng(4)

    def solve(count):
        c = b2p.Context(0)
        try:
            c.batch_upload([(s.m, s.n, s.rowptr, s.colidx, s.vals)], np.zeros(count, np.int32), np.tile(s.b, count),
                           rng.uniform(-1.0, 1.0, count * s.n), np.tile(s.lb, count), np.tile(s.ub, count),
                           np.tile(s.is_eq, count))
            if not learned:
                return c.batch_solve(precision="fp32", eps=1e-4, max_iterations=512)[0]
            c.mlp_create(8, 8, s.n + s.m + 1, seed=1)
            c.mlp_set_normalization(*[f(k, np.float32) for k in (8, s.n + s.m + 1) for f in (np.zeros, np.ones)])
            # few iterations warm, so that most instances fall back to a second, cold run
            return c.batch_solve_learned(np.ones((count, 8), np.float32), precision="fp32", eps=1e-4, max_iterations=512)[0]
        finally:
            c.close()

    for count, ni in ((600, 4), (40, 1)):
        cache.unlink(missing_ok=True)
        solve(count)
        key, threads, chunk, w, _, *forms = cache.read_text().split()
        # forms: CTA size and us per round of 1, 2 and 4 instances per CTA; four made the fastest
        forms = [forms[0], "100", forms[2], "100", forms[4], "1"]
        assert int(forms[4]) > 0
        cache.write_text(" ".join([key, forms[4], chunk, w, "4", *forms]) + "\n")
        summ = solve(count)
        assert int(round(summ["used_average"])) == 10 * ni + int(w)
        assert int(round(summ["step_size"])) // 100000 == int(forms[4])
