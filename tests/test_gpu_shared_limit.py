"""Walks whose values fill 48 KB of shared memory to the byte, beside the kernel's own
static words. FP64 <= 1e-12 relative to the oracle (max norm), FP32 <= 1e-5, refinement
<= 1e-10."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def relerr(x, ref):
    x, ref = np.asarray(x, np.float64).ravel(), np.asarray(ref, np.float64).ravel()
    return float(np.max(np.abs(x - ref)) / max(np.max(np.abs(ref)), 1e-300))


@pytest.mark.parametrize("block, rhs, dtype", [(2048, 3, np.float64), (1024, 6, np.float64), (2047, 3, np.float64),
                                               (2049, 3, np.float64), (4096, 3, np.float32), (1536, 8, np.float32)])
def test_blocked_walk_at_the_default_limit(cuda, oracle_port, block, rhs, dtype):
    from sptrsv_gb300 import SyncFreeSolver, matgen
    m = matgen.chain(9000)
    b = np.random.default_rng(rhs).standard_normal((m.n, rhs))
    ref = oracle_port.solve(m.col_ptr, m.row_idx, m.val, m.n, m.substitution, b)
    t = m.transpose()
    tref = oracle_port.solve(t.col_ptr, t.row_idx, t.val, m.n, t.substitution, b)
    s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val, order_block=block)
    x = cuda.from_numpy(b.astype(dtype)).cuda()
    tol = 1e-12 if dtype == np.float64 else 1e-5
    assert relerr(s.solve(x).cpu().numpy(), ref) <= tol
    assert relerr(s.solve_adjoint(x)[0].cpu().numpy(), tref) <= tol
    if dtype == np.float64:
        assert relerr(s.solve_refine(x)[0].cpu().numpy(), ref) <= 1e-10
    s.close()
