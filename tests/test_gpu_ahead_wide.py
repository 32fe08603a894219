"""Wide levels, where the staged-ahead walk takes one, two or three CTAs per SM by the work
per level and the length of the lists. FP64 <= 1e-12 relative to the oracle (max norm),
FP32 <= 1e-5."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def relerr(x, ref):
    x, ref = np.asarray(x, np.float64).ravel(), np.asarray(ref, np.float64).ravel()
    return float(np.max(np.abs(x - ref)) / max(np.max(np.abs(ref)), 1e-300))


@pytest.mark.parametrize("lower", [True, False])
@pytest.mark.parametrize("n, mean", [(120_000, 4.0), (400_001, 4.0), (400_000, 6.0), (250_000, 9.0), (200_003, 20.0),
                                     (600_000, 6.0)])
def test_wide_levels_match_the_oracle(cuda, oracle_port, n, mean, lower):
    from sptrsv_gb300 import SyncFreeSolver, matgen
    m = matgen.poisson_band(n, mean, n // 3, seed=n, lower=lower)
    b = np.random.default_rng(n).standard_normal(n)
    ref = oracle_port.solve(m.col_ptr, m.row_idx, m.val, n, m.substitution, b)
    t = m.transpose()
    tref = oracle_port.solve(t.col_ptr, t.row_idx, t.val, n, t.substitution, b)
    for dtype, tol in ((np.float64, 1e-12), (np.float32, 1e-5)):
        s = SyncFreeSolver(m.col_ptr, m.row_idx, n, m.substitution, values=m.val.astype(dtype))
        x = cuda.from_numpy(b.astype(dtype)).cuda()
        assert relerr(s.solve(x).cpu().numpy(), ref) <= tol
        assert relerr(s.solve_adjoint(x)[0].cpu().numpy(), tref) <= tol
        s.close()
