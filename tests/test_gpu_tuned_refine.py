"""Refinement under explicit settings that lead plain solves to the executors with lists
staged ahead (what the tuner sets), on tuned handles and on handles given such settings.
Refinement <= 1e-10 relative to the oracle (max norm), the solve itself <= 1e-12."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LEVEL_ORDER = dict(schedule=2, staged=False, warp_sync=True, order_block=2**31 - 1, backoff_ns=0, block=256)


def relerr(x, ref):
    x, ref = np.asarray(x, np.float64).ravel(), np.asarray(ref, np.float64).ravel()
    return float(np.max(np.abs(x - ref)) / max(np.max(np.abs(ref)), 1e-300))


def _matrix(kind):
    from sptrsv_gb300 import matgen
    return {"band": lambda: matgen.poisson_band(12_001, 7.0, 1500, seed=3, lower=False),
            "mesh": lambda: matgen.laplace2d_lower(150), "chain": lambda: matgen.chain(700)}[kind]()


@pytest.mark.parametrize("kind", ["band", "mesh", "chain"])
@pytest.mark.parametrize("rhs, kw", [(1, dict(chunk=256, ctas_per_sm=1, wsync_batch=1, split=0, cluster=0)),
                                     (1, dict(chunk=256, ctas_per_sm=1, split=0, cluster=1)),
                                     (2, dict(ctas_per_sm=0)), (4, dict(ctas_per_sm=0)), (15, dict(ctas_per_sm=0)),
                                     (16, dict(ctas_per_sm=0)), (33, dict(ctas_per_sm=0)), (64, dict(ctas_per_sm=0))])
def test_explicit_settings_refine(cuda, oracle_port, kind, rhs, kw):
    from sptrsv_gb300 import SyncFreeSolver
    m = _matrix(kind)
    b = np.random.default_rng(rhs).standard_normal((m.n, rhs))
    ref = oracle_port.solve(m.col_ptr, m.row_idx, m.val, m.n, m.substitution, b)
    s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val, **LEVEL_ORDER, **kw)
    x = cuda.from_numpy(b).cuda()
    for layout in (x, x.t().contiguous().t()):
        assert relerr(s.solve(layout).cpu().numpy(), ref) <= 1e-12
        assert relerr(s.solve_refine(layout)[0].cpu().numpy(), ref) <= 1e-10
        assert relerr(s.solve_refine(layout, tol=0.0, max_iter=2)[0].cpu().numpy(), ref) <= 1e-10
    s.close()


@pytest.mark.parametrize("rhs", [1, 4, 16])
@pytest.mark.parametrize("kind", ["band", "mesh", "batch"])
def test_tuned_handles_refine(cuda, oracle_port, kind, rhs):
    from sptrsv_gb300 import SyncFreeSolver, matgen
    ms = matgen.batch_uneven(count=6, seed=2, nmin=200, nmax=6000) if kind == "batch" else [_matrix(kind)]
    bs = [np.random.default_rng(i).standard_normal((m.n, rhs)) for i, m in enumerate(ms)]
    ref = np.concatenate([oracle_port.solve(m.col_ptr, m.row_idx, m.val, m.n, m.substitution, b).reshape(m.n, rhs)
                          for m, b in zip(ms, bs)])
    val = np.concatenate([m.val for m in ms])
    if kind == "batch":
        s = SyncFreeSolver(batch=[(m.col_ptr, m.row_idx, m.n, m.substitution) for m in ms], values=val)
    else:
        s = SyncFreeSolver(ms[0].col_ptr, ms[0].row_idx, ms[0].n, ms[0].substitution, values=val)
    x = cuda.from_numpy(np.concatenate(bs)).cuda()
    s.tune(x, reps=2)
    assert relerr(s.solve(x).cpu().numpy(), ref) <= 1e-12
    assert relerr(s.solve_refine(x)[0].cpu().numpy(), ref) <= 1e-10
    s.close()
