"""Level-order executor with lists staged ahead for several right-hand sides: every lane
shape (1, 2 or 4 right-hand sides per lane, odd and even counts around its limits), sizes
around its chunks, both layouts, directions and precisions. FP64 <= 1e-12 relative
against the oracle (max norm, the tolerance of every pull executor), FP32 <= 1e-5."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def relerr(x, ref):
    x, ref = np.asarray(x, np.float64), np.asarray(ref, np.float64)
    return float(np.max(np.abs(x - ref)) / max(np.max(np.abs(ref)), 1e-300))


def _check(cuda, oracle_port, m, rhs, col_major, **kw):
    from sptrsv_gb300 import SyncFreeSolver
    rng = np.random.default_rng(m.n + rhs)
    b = rng.standard_normal((m.n, rhs))
    ref = oracle_port.solve(m.col_ptr, m.row_idx, m.val, m.n, m.substitution, b)
    t = m.transpose()
    tref = oracle_port.solve(t.col_ptr, t.row_idx, t.val, m.n, t.substitution, b)
    for dtype, tol in ((np.float64, 1e-12), (np.float32, 1e-5)):
        s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val.astype(dtype), **kw)
        bd = cuda.from_numpy(b.astype(dtype)).cuda()
        if col_major:
            bd = bd.t().contiguous().t()
        for _ in range(2):   # the ticket starts over
            assert relerr(s.solve(bd).cpu().numpy(), ref) <= tol
            assert relerr(s.solve_adjoint(bd)[0].cpu().numpy(), tref) <= tol
        s.close()


@pytest.mark.parametrize("lower", [True, False])
@pytest.mark.parametrize("rhs", [2, 3, 4, 5, 8, 9, 10, 16, 17, 18, 31, 32, 33, 34, 62, 63, 64])
def test_every_lane_shape(cuda, oracle_port, rhs, lower):
    from sptrsv_gb300 import matgen
    m = matgen.poisson_band(5001, 7.0, 1500, seed=rhs, lower=lower)
    _check(cuda, oracle_port, m, rhs, col_major=bool(rhs % 3))


@pytest.mark.parametrize("rhs", [2, 8, 16, 64])
@pytest.mark.parametrize("kind, n", [("band", 1), ("band", 7), ("band", 8), ("band", 127), ("band", 129),
                                     ("chain", 300), ("dense", 300), ("diagonal", 1000), ("wide", 60_000)])
def test_sizes_around_the_chunks(cuda, oracle_port, kind, n, rhs):
    """Chunks of 8 to 128 unknowns, chains inside a chunk, lists past its buffer (dense), levels past 350 unknowns
    (wide: pairs per lane at 16 right-hand sides)."""
    from sptrsv_gb300 import matgen
    m = {"band": lambda: matgen.poisson_band(n, 6.0, max(n // 2, 2), seed=n), "chain": lambda: matgen.chain(n),
         "dense": lambda: matgen.dense_lower(n), "diagonal": lambda: matgen.diagonal(n),
         "wide": lambda: matgen.poisson_band(n, 3.0, n // 2, seed=n)}[kind]()
    _check(cuda, oracle_port, m, rhs, col_major=False, order_block=2**31 - 1)


@pytest.mark.parametrize("rhs", [9, 15, 17, 31, 33, 35, 63])
def test_counts_that_are_not_whole_lanes(cuda, oracle_port, rhs):
    """Levels past 350 unknowns; the values around the solution block stay as they are."""
    from sptrsv_gb300 import SyncFreeSolver, matgen
    m = matgen.poisson_band(20_001, 3.0, 10_000, seed=rhs)
    _check(cuda, oracle_port, m, rhs, col_major=rhs % 4 == 1, order_block=2**31 - 1)
    b = np.random.default_rng(rhs).standard_normal((m.n, rhs))
    ref = oracle_port.solve(m.col_ptr, m.row_idx, m.val, m.n, m.substitution, b)
    s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val, order_block=2**31 - 1)
    room = cuda.full((m.n + 2, rhs), 7.0, dtype=cuda.float64, device="cuda")
    bd = cuda.from_numpy(b).cuda()
    s.solve(bd, out=room[1:-1])
    assert relerr(room[1:-1].cpu().numpy(), ref) <= 1e-12
    s.solve_refine(bd, out=room[1:-1])
    assert relerr(room[1:-1].cpu().numpy(), ref) <= 1e-10
    assert bool((room[0] == 7.0).all()) and bool((room[-1] == 7.0).all())
    s.close()


def test_infinities_and_nan_stay_in_their_column(cuda):
    """Against the executor with an explicit right-hand-side tile."""
    from sptrsv_gb300 import SyncFreeSolver, matgen
    m = matgen.poisson_band(3001, 6.0, 800, seed=4)
    for rhs in (8, 16, 64):
        b = np.random.default_rng(rhs).standard_normal((m.n, rhs))
        b[7, 0], b[500, rhs - 1] = np.inf, -np.inf
        b.view(np.uint64)[1200, 1] = 0xFFFFFFFFFFFFFFFF
        out = []
        for kw in (dict(rhs_tile=2), dict()):
            s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val, **kw)
            out.append(s.solve(cuda.from_numpy(b).cuda()).cpu().numpy())
        assert np.array_equal(np.isnan(out[0]), np.isnan(out[1]))
        assert np.array_equal(np.isinf(out[0]), np.isinf(out[1]))
        ok = np.isfinite(out[0])
        assert relerr(out[1][ok], out[0][ok]) <= 1e-12


@pytest.mark.parametrize("rhs", [1, 2, 4, 7, 8, 15, 16, 18, 31, 32, 34, 63, 64])
@pytest.mark.parametrize("kind, n", [("band", 33), ("band", 5001), ("chain", 300), ("dense", 300), ("wide", 60_000)])
def test_refined_blocks(cuda, oracle_port, kind, n, rhs):
    """The fused first refinement step over the same lane shapes (1e-10, the refinement's tolerance)."""
    from sptrsv_gb300 import SyncFreeSolver, matgen
    m = {"band": lambda: matgen.poisson_band(n, 7.0, max(n // 3, 2), seed=n), "chain": lambda: matgen.chain(n),
         "dense": lambda: matgen.dense_lower(n), "wide": lambda: matgen.poisson_band(n, 3.0, n // 2, seed=n)}[kind]()
    b = np.random.default_rng(rhs).standard_normal((m.n, rhs))
    ref = oracle_port.solve(m.col_ptr, m.row_idx, m.val, m.n, m.substitution, b)
    s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val)
    bd = cuda.from_numpy(b).cuda()
    for _ in range(2):
        x, iters, est = s.solve_refine(bd)
        assert 1 <= iters <= 4 and est <= 1e-12
        assert relerr(x.cpu().numpy(), ref) <= 1e-10


@pytest.mark.parametrize("rhs", [2, 5, 16, 31, 32])
def test_refined_columns(cuda, oracle_port, rhs):
    """Column-major blocks through the fused step as they are (below 32), further steps on rows: a tolerance that one
    step (FP32, about 1e-14 by the estimate) does not reach; the solution over its right-hand side."""
    from sptrsv_gb300 import SyncFreeSolver, matgen
    m = matgen.poisson_band(20_001, 3.0, 10_000, seed=rhs)
    b = np.random.default_rng(rhs).standard_normal((m.n, rhs))
    ref = oracle_port.solve(m.col_ptr, m.row_idx, m.val, m.n, m.substitution, b)
    s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val)
    bd = cuda.from_numpy(b).cuda().t().contiguous().t()
    x, iters, est = s.solve_refine(bd, tol=1e-12)
    assert iters == 1 and relerr(x.cpu().numpy(), ref) <= 1e-10
    for tol, want in ((1e-18, 2), (0.0, 3)):
        x, iters, _ = s.solve_refine(bd, tol=tol, max_iter=3 if tol == 0.0 else 10)
        assert iters >= want
        assert relerr(x.cpu().numpy(), ref) <= 1e-12
    s.solve_refine(bd, tol=1e-18, out=bd)
    assert relerr(bd.cpu().numpy(), ref) <= 1e-12
    s.close()
