"""Values and captured graphs: whatever a graph reads or stages, its replays and the calls
between them use the current values. FP64 <= 1e-12 and FP32 <= 1e-5 relative to the oracle
(max norm), refinement <= 1e-10, as in the executors' own tests."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def relerr(x, ref):
    x, ref = np.asarray(x, np.float64).ravel(), np.asarray(ref, np.float64).ravel()
    return float(np.max(np.abs(x - ref)) / max(np.max(np.abs(ref)), 1e-300))


@pytest.fixture
def own_stream(cuda):
    with cuda.cuda.stream(cuda.cuda.Stream()):
        yield
        cuda.cuda.current_stream().synchronize()


def _band(n, lower=True):
    from sptrsv_gb300 import matgen
    return matgen.poisson_band(n, 5.0, max(n // 5, 2), seed=n, lower=lower)


@pytest.mark.parametrize("n", [1, 33, 3000])
def test_captured_staging_follows_values_of_either_precision(cuda, oracle_port, own_stream, n):
    """A graph that stages the transposed FP32 weights itself (their first use is inside the
    capture), replayed after values of the other precision were set."""
    from sptrsv_gb300 import SyncFreeSolver
    m = _band(n)
    rng = np.random.default_rng(n)
    b = rng.standard_normal(m.n)
    stream = cuda.cuda.current_stream()
    bf = cuda.from_numpy(b.astype(np.float32)).cuda()
    lam = cuda.empty_like(bf)
    s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val.astype(np.float32), sync_check=False,
                       stream=stream)
    s.solve(bf)
    stream.synchronize()
    g = cuda.cuda.CUDAGraph()
    with cuda.cuda.graph(g, stream=stream):
        s.solve_adjoint(bf, out=lam)
    for dtype in (np.float32, np.float64, np.float32, np.float64):
        val = (m.val * rng.uniform(0.9, 1.1, m.nnz)).astype(dtype)
        s.set_values(val)
        lam.zero_()
        g.replay()
        t = type(m)(m.n, m.col_ptr, m.row_idx, val.astype(np.float64), m.lower).transpose()
        ref = oracle_port.solve(t.col_ptr, t.row_idx, t.val, m.n, t.substitution, b)
        assert relerr(lam.cpu().numpy(), ref) <= 1e-5
    s.check()
