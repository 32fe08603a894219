"""sptrsv_info.wsync_batch: list entries per lane and iteration of the executor that runs
the forward walk (wide levels poll two entries at once, a cluster one, one consumer per
block takes whole lists)."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind, kw, want", [("wide", dict(), 2), ("wide", dict(wsync_batch=1), 1), ("narrow", dict(), 1),
                                            ("narrow", dict(cluster=0), 1), ("long mesh", dict(), 2),
                                            ("four", dict(), 4), ("wide", dict(block=128), 1)])
def test_entries_per_iteration_of_the_executor_in_use(cuda, kind, kw, want):
    import numpy as np
    from sptrsv_gb300 import SyncFreeSolver, matgen
    m = {"wide": lambda: matgen.poisson_band(500_000, 9.0, 150_000, seed=1),
         "narrow": lambda: matgen.poisson_band(10_000, 8.0, 2000, seed=1),
         "long mesh": lambda: matgen.laplace2d_lower(150),
         "four": lambda: matgen.banded_random_lower(4000, np.full(4000, 4), 60, 1, lower=False)}[kind]()
    if kind == "four":   # rows of at most four entries in blocks of 300
        kw = dict(schedule=2, staged=False, warp_sync=True, order_block=300, chunk=300, block=128, ctas_per_sm=0,
                  backoff_ns=0, split=0)
    s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val, **kw)
    assert s.info()["wsync_batch"] == want
    s.solve(cuda.ones(m.n, dtype=cuda.float64, device="cuda"))
    assert s.info()["wsync_batch"] == want
    s.close()
