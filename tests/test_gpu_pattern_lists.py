"""Analysis of list lengths around the limits of the sync-free level pass (256
dependencies) and of the rank-sorted lists (1,024 entries):
CSR exactly the transposed pattern, level sets and in-degree exact, and solves that walk
the sorted lists in both directions (FP64 <= 1e-12 relative, max norm)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lower", [True, False])
@pytest.mark.parametrize("kind, n", [("star", 2), ("star", 33), ("star", 257), ("star", 258), ("star", 1024), ("star", 1025), ("star", 1026),
                                     ("dense", 65), ("band", 1), ("band", 31), ("band", 4097), ("diagonal", 100)])
def test_lists_around_the_rank_limit(cuda, oracle_port, kind, n, lower):
    from sptrsv_gb300 import SyncFreeSolver, matgen
    m = {"star": lambda: matgen.star(n, lower=lower), "dense": lambda: matgen.dense_lower(n, lower=lower),
         "band": lambda: matgen.poisson_band(n, 9.0, max(n // 2, 2), seed=n, lower=lower),
         "diagonal": lambda: matgen.diagonal(n, lower=lower)}[kind]()
    s = SyncFreeSolver(m.col_ptr, m.row_idx, n, m.substitution, values=m.val)
    t = m.transpose()
    rp, ci, src = (a.cpu().numpy() for a in s.csr())
    assert np.array_equal(rp, t.col_ptr) and np.array_equal(ci, t.row_idx)
    assert np.array_equal(m.val[src], t.val)
    inf = s.info()
    assert inf["max_in_degree"] == int(np.max(np.diff(t.col_ptr)))
    depth = np.zeros(n, np.int64)
    for i in (range(n) if lower else range(n - 1, -1, -1)):
        deps = ci[rp[i]:rp[i + 1]]
        deps = deps[deps != i]
        depth[i] = depth[deps].max() + 1 if deps.size else 0
    lp, li = (a.cpu().numpy() for a in s.levels())
    assert inf["nlevels"] == depth.max() + 1
    assert np.array_equal(lp, np.concatenate([[0], np.cumsum(np.bincount(depth))]))
    assert np.array_equal(li, np.lexsort((np.arange(n), depth)))
    b = np.random.default_rng(n).standard_normal(n)
    for x, tri in ((s.solve(cuda.from_numpy(b).cuda()), m), (s.solve_adjoint(cuda.from_numpy(b).cuda())[0], t)):
        ref = oracle_port.solve(tri.col_ptr, tri.row_idx, tri.val, n, tri.substitution, b)
        assert np.max(np.abs(x.cpu().numpy() - ref)) <= 1e-12 * np.max(np.abs(ref))
