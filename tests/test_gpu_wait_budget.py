"""The wait budget bounds a wait, not the work: one list that takes several budgets to
walk although all its entries were published early. FP64 <= 1e-12 relative to the oracle
(max norm), refinement <= 1e-10."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def relerr(x, ref):
    x, ref = np.asarray(x, np.float64).ravel(), np.asarray(ref, np.float64).ravel()
    return float(np.max(np.abs(x - ref)) / max(np.max(np.abs(ref)), 1e-300))


def _long_list(length, others, chain, seed):
    """Lower triangle: unknowns 1 .. chain - 1 follow one another, `others` hang on one or
    two of them, and the last unknown depends on `length` of those."""
    from sptrsv_gb300 import matgen
    rng = np.random.default_rng(seed)
    n = chain + others + 1
    row = np.arange(chain, chain + others)
    rows = np.concatenate([np.arange(1, chain), row, row, np.full(length, n - 1)])
    cols = np.concatenate([np.arange(chain - 1), rng.integers(0, chain, others),
                           rng.integers(0, chain, others), chain + np.arange(length)])
    key = np.unique(cols.astype(np.int64) * n + rows)
    return matgen._explicit_lower(n, key // n, key % n, seed, True)


# lists of one lane, 50,000 entries and more (at ~0.2 us each, ten budgets), and of 32 lanes
# that hold 20,000 each
@pytest.mark.parametrize("call, rhs, length, others, chain, kw", [
    ("solve", 1, 60_000, 60_000, 2, dict(split=0, cluster=0)),
    ("solve", 1, 60_000, 60_000, 2, dict(cluster=1)),
    ("solve", 1, 640_000, 640_000, 400, dict(cluster=0)),
    ("solve", 2, 50_000, 700_000, 2, dict()),
    ("solve", 16, 50_000, 700_000, 2, dict()),
    ("refine", 1, 60_000, 60_000, 2, dict(split=0)),
    ("refine", 8, 50_000, 700_000, 2, dict())])
def test_a_long_list_is_no_long_wait(cuda, oracle_port, call, rhs, length, others, chain, kw):
    from sptrsv_gb300 import SyncFreeSolver, _lib
    m = _long_list(length, others, chain, 7)
    b = np.random.default_rng(rhs).standard_normal((m.n, rhs))
    ref = oracle_port.solve(m.col_ptr, m.row_idx, m.val, m.n, m.substitution, b)
    s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val, order_block=2**31 - 1, **kw)
    s.set_option(_lib.OPTION_TIMEOUT_MS, 1)
    bd = cuda.from_numpy(b).cuda()
    x = s.solve(bd) if call == "solve" else s.solve_refine(bd)[0]
    assert relerr(x.cpu().numpy(), ref) <= (1e-12 if call == "solve" else 1e-10)
    s.close()
