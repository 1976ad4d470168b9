"""What a reference solve leaves on the device."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


def test_large_solve_gives_its_buffers_back(b2p, lpgen):
    """The sliced copies of a large LP are as large as the LP; only the LP itself stays with the context."""
    import torch
    c = b2p.Context(0)
    try:
        c.upload(lpgen.random_sparse(m=9000, n=30000, nnz_per_col=3, seed=1).standard())
        c.solve(engine="reference", max_iterations=100)  # kernels are loaded
        c.upload(lpgen.random_sparse(m=100000, n=400000, nnz_per_col=6, seed=1).standard())
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        for _ in range(2):
            r, _, _ = c.solve(engine="reference", max_iterations=100)
            assert r["iterations"] == 100
        # the copies alone are 2 * 12 bytes for each of 2.4 million entries
        assert before - torch.cuda.mem_get_info()[0] < 16 << 20
    finally:
        c.close()
