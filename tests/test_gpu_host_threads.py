"""Contexts on several host threads.  How much dynamic shared memory a kernel may be launched with is
state of the function, shared by all of them: no call may lower it for another one."""
from __future__ import annotations

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROUNDS = 150
# per thread: LPs of different sizes, so that the threads need different amounts at any time
SIZES = [[(60, 200, 4), (1500, 4500, 6)], [(1200, 4000, 5), (40, 130, 3)], [(300, 1000, 5), (900, 3000, 4)], [(700, 2500, 5), (280, 900, 4)]] * 2


def call(c, kind, s):
    if kind == "reference":
        c.upload(s)
        r, x, y = c.solve(engine="reference", max_iterations=60)
    elif kind == "halpern":
        c.upload(s)
        r, x, y = c.solve(engine="halpern", precision="fp64", eps=0.0, max_iterations=64)
    elif kind == "spmv_t":
        w, _ = c.spmv(s.m, s.n, s.rowptr, s.colidx, s.vals, s.b, transpose=True)
        return [w]
    else:
        c.batch_upload([(s.m, s.n, s.rowptr, s.colidx, s.vals)] * 3, np.arange(3, dtype=np.int32),
                       *[np.tile(v, 3) for v in (s.b, s.c, s.lb, s.ub, s.is_eq)])
        _, _, x, y = c.batch_solve(precision="fp64", eps=1e-14, max_iterations=128, check_every=64)
    return [x, y]


@pytest.mark.parametrize("kind", ["reference", "halpern", "spmv_t", "batch"])
def test_threads_do_not_disturb_each_other(b2p, lpgen, tmp_path, monkeypatch, kind):
    """Every call of every thread succeeds and gives what one thread alone gets: bit for bit, except the
    single-LP engine, whose sums of squares are added in any order (256 * 20 * 2^-53 of the norm)."""
    monkeypatch.setenv("B2P_AUTOTUNE_CACHE", str(tmp_path / "tune.txt"))
    lps = [[lpgen.random_sparse(m=m, n=n, nnz_per_col=k, seed=m).standard() for m, n, k in t] for t in SIZES]
    alone = b2p.Context(0)
    try:
        want = [[call(alone, kind, s) for s in t] for t in lps]
    finally:
        alone.close()
    wrong = []
    start = threading.Barrier(len(lps))

    def work(t):
        c = b2p.Context(0)
        try:
            start.wait()
            for _ in range(ROUNDS):
                for s, w in zip(lps[t], want[t]):
                    for a, b in zip(call(c, kind, s), w):
                        same = np.array_equal(a, b) if kind != "halpern" else (
                            np.linalg.norm(a - b) <= 1e-10 * (1 + np.linalg.norm(b)))
                        if not same:
                            wrong.append((t, s.m, float(np.abs(a - b).max())))
        except Exception as e:  # noqa: BLE001  (reported below, outside the thread)
            wrong.append((t, repr(e)))
        finally:
            c.close()

    threads = [threading.Thread(target=work, args=(t,)) for t in range(len(lps))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:4]
