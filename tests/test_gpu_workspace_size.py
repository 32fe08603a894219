"""Calls with one number of right-hand sides and one type use workspaces of one size,
whichever executor pads its rows: a graph captured from one call keeps its buffers when
another runs outside it."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rhs", [7, 9, 15, 31, 33, 61, 63])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_one_size_per_count_and_type(cuda, rhs, dtype):
    from sptrsv_gb300 import SyncFreeSolver, matgen
    m = matgen.poisson_band(3000, 5.0, 900, seed=rhs)
    s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val.astype(dtype))
    one = cuda.from_numpy(np.random.default_rng(rhs).standard_normal((m.n, rhs)).astype(dtype)).cuda()
    s.solve(one[:, 0].contiguous())
    s.solve_adjoint(one[:, 0].contiguous())    # both directions' weights are staged
    s.solve_adjoint(one)
    size = s.info()["device_bytes"]
    s.solve(one)
    assert s.info()["device_bytes"] == size
    s.solve(one.t().contiguous().t())          # the copies of column-major blocks
    size = s.info()["device_bytes"]
    for x in (one, one.t().contiguous().t()):
        s.solve(x)
        s.solve_adjoint(x)
    assert s.info()["device_bytes"] == size
    s.close()
