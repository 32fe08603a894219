"""Gradient with respect to the values, rows read 16 bytes at a time where they allow it:
counts around whole 16-byte words, both layouts and precisions, rows that start off a
16-byte boundary. Against the sum in FP64: n sums of at most 64 products, FP64 <= 1e-13
and FP32 <= 1e-5 relative (max norm)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("col_major", [False, True])
@pytest.mark.parametrize("rhs", [1, 4, 7, 8, 9, 10, 12, 16, 64])
def test_grad_values(cuda, rhs, col_major, offset):
    from sptrsv_gb300 import SyncFreeSolver, matgen
    m = matgen.poisson_band(2001, 5.0, 300, seed=rhs)
    cols = np.repeat(np.arange(m.n), np.diff(m.col_ptr))
    rng = np.random.default_rng(rhs)
    for dtype, tol in ((np.float64, 1e-13), (np.float32, 1e-5)):
        s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val.astype(dtype))
        a, b = (rng.standard_normal((m.n, rhs)).astype(dtype) for _ in range(2))
        views = []
        for v in (a, b):
            room = cuda.zeros(m.n * rhs + 4, dtype=cuda.from_numpy(v).dtype, device="cuda")
            flat = room[offset:offset + m.n * rhs]
            t = flat.view(rhs, m.n).t() if col_major else flat.view(m.n, rhs)
            t.copy_(cuda.from_numpy(v))
            views.append(t)
        got = s.grad_values(*views).cpu().numpy()
        want = -(a.astype(np.float64)[m.row_idx] * b.astype(np.float64)[cols]).sum(1)
        assert np.max(np.abs(got - want)) <= tol * np.max(np.abs(want))
        s.close()
