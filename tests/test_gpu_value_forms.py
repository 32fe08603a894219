"""Staged value forms: every executor stages the forms it needs when it first runs, and
new values reach all of them. FP64 <= 1e-12 and FP32 <= 1e-5 relative to the oracle
(max norm), refinement <= 1e-10, as in the executors' own tests."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def relerr(x, ref):
    x, ref = np.asarray(x, np.float64).ravel(), np.asarray(ref, np.float64).ravel()
    return float(np.max(np.abs(x - ref)) / max(np.max(np.abs(ref)), 1e-300))


def _check_all(cuda, oracle_port, s, m, val, b, f64=True):
    from sptrsv_gb300 import _lib
    ref = oracle_port.solve(m.col_ptr, m.row_idx, val, m.n, m.substitution, b)
    t = type(m)(m.n, m.col_ptr, m.row_idx, val, m.lower).transpose()
    tref = oracle_port.solve(t.col_ptr, t.row_idx, t.val, m.n, t.substitution, b)
    bd, bf = cuda.from_numpy(b).cuda(), cuda.from_numpy(b.astype(np.float32)).cuda()
    got = {}
    if f64:
        got["solve"] = (s.solve(bd), ref, 1e-12)
        got["adjoint"] = (s.solve_adjoint(bd)[0], tref, 1e-12)
        got["refine"] = (s.solve_refine(bd)[0], ref, 1e-10)
        for name, opt, v in (("exact", _lib.OPTION_EXACT, 1), ("push", _lib.OPTION_SCHEDULE, 1)):
            old = s.get_option(opt)
            s.set_option(opt, v)
            got[name] = (s.solve(bd), ref, 1e-12)
            if name == "exact":
                got["exact adjoint"] = (s.solve_adjoint(bd)[0], tref, 1e-12)
            s.set_option(opt, old)
    got["solve f32"] = (s.solve(bf), ref, 1e-5)
    got["adjoint f32"] = (s.solve_adjoint(bf)[0], tref, 1e-5)
    for name, (x, r, tol) in got.items():
        assert relerr(x.cpu().numpy(), r) <= tol, name


@pytest.mark.parametrize("lower", [True, False])
@pytest.mark.parametrize("n, mean", [(1, 0.0), (33, 3.0), (700, 0.0), (5003, 7.0), (20_000, 2.0)])
def test_new_values_reach_every_form(cuda, oracle_port, n, mean, lower):
    from sptrsv_gb300 import SyncFreeSolver, matgen
    m = matgen.poisson_band(n, mean, max(n // 3, 2), seed=n, lower=lower)
    rng = np.random.default_rng(n)
    b = rng.standard_normal(n)
    s = SyncFreeSolver(m.col_ptr, m.row_idx, n, m.substitution, values=m.val, order_block=2**31 - 1)
    _check_all(cuda, oracle_port, s, m, m.val, b)
    for step in range(2):   # the second set goes through a solve that brings its values
        val = m.val * rng.uniform(0.9, 1.1, m.nnz)
        if step:
            s.solve(cuda.from_numpy(b).cuda(), values=cuda.from_numpy(val).cuda())
        else:
            s.set_values(val)
        _check_all(cuda, oracle_port, s, m, val, b)
    val32 = (m.val * rng.uniform(0.9, 1.1, m.nnz)).astype(np.float32)
    s.set_values(val32)
    _check_all(cuda, oracle_port, s, m, val32.astype(np.float64), b, f64=False)
    s.set_values(m.val)
    _check_all(cuda, oracle_port, s, m, m.val, b)


@pytest.mark.parametrize("star_lower", [True, False])
def test_long_and_empty_lists(cuda, oracle_port, star_lower):
    """One list of 2,999 entries among empty ones: owners found across whole warps."""
    from sptrsv_gb300 import SyncFreeSolver, matgen
    m = matgen.star(3000, lower=star_lower)
    s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val)
    _check_all(cuda, oracle_port, s, m, m.val, np.random.default_rng(1).standard_normal(m.n))


def test_first_adjoint_inside_a_capture(cuda, oracle_port):
    """A form first needed while a graph is captured is staged by the graph, also for
    values set after the capture, and by the next call outside it."""
    from sptrsv_gb300 import SyncFreeSolver, matgen
    m = matgen.poisson_band(3000, 5.0, 600, seed=9)
    rng = np.random.default_rng(9)
    b = rng.standard_normal(m.n)
    stream = cuda.cuda.Stream()
    with cuda.cuda.stream(stream):
        bd = cuda.from_numpy(b).cuda()
        lam = cuda.empty_like(bd)
        s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val, sync_check=False, stream=stream)
        s.solve(bd)
        stream.synchronize()
        g = cuda.cuda.CUDAGraph()
        with cuda.cuda.graph(g, stream=stream):
            s.solve_adjoint(bd, out=lam)
        eager, _ = s.solve_adjoint(bd)
        for val in (m.val, m.val * rng.uniform(0.9, 1.1, m.nnz)):
            s.set_values(val)
            g.replay()
            stream.synchronize()
            t = type(m)(m.n, m.col_ptr, m.row_idx, val, m.lower).transpose()
            ref = oracle_port.solve(t.col_ptr, t.row_idx, t.val, m.n, t.substitution, b)
            assert relerr(lam.cpu().numpy(), ref) <= 1e-12
            if val is m.val:
                assert relerr(eager.cpu().numpy(), ref) <= 1e-12
        s.check()
