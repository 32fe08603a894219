"""Systems whose neighbouring lists are of unlike length, on levels narrow and wide enough
for either executor family: stripes of columns, and batches of unlike members. FP64 <=
1e-12 relative to the oracle (max norm), FP32 <= 1e-5, refinement <= 1e-10."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def relerr(x, ref):
    x, ref = np.asarray(x, np.float64).ravel(), np.asarray(ref, np.float64).ravel()
    return float(np.max(np.abs(x - ref)) / max(np.max(np.abs(ref)), 1e-300))


def _stripes(n, band, stripe, lower):
    from sptrsv_gb300 import matgen
    counts = np.where((np.arange(n) // stripe) % 2, 2, 18)
    return matgen.banded_random_lower(n, counts, band, n, lower=lower)


def _members(kind):
    from sptrsv_gb300 import matgen
    if kind == "narrow":
        return [_stripes(20_000, 400, 300, True)]
    if kind == "wide":
        return [_stripes(60_001, 20_000, 500, False)]
    means = (2, 18, 5, 20, 3, 12)
    return [matgen.poisson_band(7000 + 500 * i, float(k), 400 if kind == "narrow batch" else 3000, seed=i, lower=i % 2 == 0)
            for i, k in enumerate(means)]


@pytest.mark.parametrize("rhs", [1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("kind", ["narrow", "wide", "narrow batch", "wide batch"])
def test_unlike_lists_match_the_oracle(cuda, oracle_port, kind, rhs):
    from sptrsv_gb300 import SyncFreeSolver
    ms = _members(kind)
    bs = [np.random.default_rng(i).standard_normal((m.n, rhs)) for i, m in enumerate(ms)]
    ref = np.concatenate([oracle_port.solve(m.col_ptr, m.row_idx, m.val, m.n, m.substitution, b).reshape(m.n, rhs)
                          for m, b in zip(ms, bs)])
    ts = [m.transpose() for m in ms]
    tref = np.concatenate([oracle_port.solve(t.col_ptr, t.row_idx, t.val, t.n, t.substitution, b).reshape(t.n, rhs)
                           for t, b in zip(ts, bs)])
    val, b = np.concatenate([m.val for m in ms]), np.concatenate(bs)
    for dtype, tol in ((np.float64, 1e-12), (np.float32, 1e-5)):
        if len(ms) == 1:
            s = SyncFreeSolver(ms[0].col_ptr, ms[0].row_idx, ms[0].n, ms[0].substitution, values=val.astype(dtype))
        else:
            s = SyncFreeSolver(batch=[(m.col_ptr, m.row_idx, m.n, m.substitution) for m in ms], values=val.astype(dtype))
        x = cuda.from_numpy(b.astype(dtype)).cuda()
        for layout in (x, x.t().contiguous().t()):
            assert relerr(s.solve(layout).cpu().numpy(), ref) <= tol
            assert relerr(s.solve_adjoint(layout)[0].cpu().numpy(), tref) <= tol
            if dtype == np.float64:
                assert relerr(s.solve_refine(layout)[0].cpu().numpy(), ref) <= 1e-10
        s.close()
