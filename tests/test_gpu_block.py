"""Blocked layouts: the one-consumer walk of a unit's level segments and the unit and
import tables built on the device. Units around a segment (32 positions), the ring (16
segments), ragged last units, levels of one and of several segments, lists of one to four
entries, both precisions and directions, several systems in one handle. FP64 <= 1e-12
relative against the oracle (max norm, the tolerance of every pull executor), FP32 <= 1e-5.
wsync_batch=1 asks for the importer executor, whose tables serve lists of any length."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def relerr(x, ref):
    x, ref = np.asarray(x, np.float64).ravel(), np.asarray(ref, np.float64).ravel()
    return float(np.max(np.abs(x - ref)) / max(np.max(np.abs(ref)), 1e-300))


def _matrix(kind, n, lower):
    from sptrsv_gb300 import matgen
    if kind.startswith("lists"):   # the transpose's columns become lists of at most that many entries
        counts = np.random.default_rng(n).integers(0, int(kind[5:]) + 1, size=n)
        counts[0] = int(kind[5:])
        return matgen.banded_random_lower(n, counts, 60, n, lower=lower)
    return {"chain": lambda: matgen.chain(n, lower=lower), "mesh": lambda: matgen.laplace2d_lower(n, lower=lower),
            "band": lambda: matgen.poisson_band(n, 7.0, 40, seed=n, lower=lower)}[kind]()


def _blocked(block):
    return dict(schedule=2, staged=False, warp_sync=True, order_block=block, chunk=block, block=128, ctas_per_sm=0,
                backoff_ns=0, split=0)


@pytest.mark.parametrize("batch", [None, 1])
@pytest.mark.parametrize("block", [31, 32, 33, 513, 2000])
@pytest.mark.parametrize("kind, n, lower", [("chain", 700, True), ("mesh", 40, True), ("mesh", 67, False),
                                            ("lists1", 3001, False), ("lists3", 4000, False),
                                            ("lists4", 4001, False), ("band", 3000, True)])
def test_blocked_solves_match_the_oracle(cuda, oracle_port, kind, n, lower, block, batch):
    from sptrsv_gb300 import SyncFreeSolver
    m = _matrix(kind, n, lower)
    b = np.random.default_rng(n).standard_normal(m.n)
    ref = oracle_port.solve(m.col_ptr, m.row_idx, m.val, m.n, m.substitution, b)
    t = m.transpose()
    tref = oracle_port.solve(t.col_ptr, t.row_idx, t.val, m.n, t.substitution, b)
    kw = _blocked(min(block, m.n - 1))
    if batch:
        kw["wsync_batch"] = batch
    for dtype, tol in ((np.float64, 1e-12), (np.float32, 1e-5)):
        s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val.astype(dtype), **kw)
        x = cuda.from_numpy(b.astype(dtype)).cuda()
        for _ in range(2):
            assert relerr(s.solve(x).cpu().numpy(), ref) <= tol
            assert relerr(s.solve_adjoint(x)[0].cpu().numpy(), tref) <= tol
        s.solve(x, out=x)   # in place
        assert relerr(x.cpu().numpy(), ref) <= tol
        s.close()


@pytest.mark.parametrize("grid, lower", [(150, True), (190, False)])
def test_automatic_plan_of_a_mesh(cuda, oracle_port, grid, lower):
    from sptrsv_gb300 import SyncFreeSolver
    m = _matrix("mesh", grid, lower)
    b = np.random.default_rng(grid).standard_normal(m.n)
    ref = oracle_port.solve(m.col_ptr, m.row_idx, m.val, m.n, m.substitution, b)
    t = m.transpose()
    tref = oracle_port.solve(t.col_ptr, t.row_idx, t.val, m.n, t.substitution, b)
    for dtype, tol in ((np.float64, 1e-12), (np.float32, 1e-5)):
        s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val.astype(dtype), cluster=0)
        assert s.info()["order_block"] < m.n
        x = cuda.from_numpy(b.astype(dtype)).cuda()
        assert relerr(s.solve(x).cpu().numpy(), ref) <= tol
        assert relerr(s.solve_adjoint(x)[0].cpu().numpy(), tref) <= tol
        s.close()


@pytest.mark.parametrize("rhs", [8, 9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("grid, lower, col_major", [(150, True, False), (131, False, True), (400, True, False)])
def test_blocks_walk_a_mesh_in_level_order(cuda, oracle_port, grid, lower, col_major, rhs):
    """Blocks of right-hand sides on the automatic plan's blocked layout, narrow and wide levels."""
    from sptrsv_gb300 import SyncFreeSolver
    m = _matrix("mesh", grid, lower)
    b = np.random.default_rng(rhs).standard_normal((m.n, rhs))
    ref = oracle_port.solve(m.col_ptr, m.row_idx, m.val, m.n, m.substitution, b)
    t = m.transpose()
    tref = oracle_port.solve(t.col_ptr, t.row_idx, t.val, m.n, t.substitution, b)
    for dtype, tol in ((np.float64, 1e-12), (np.float32, 1e-5)):
        s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val.astype(dtype))
        assert s.info()["order_block"] < m.n
        x = cuda.from_numpy(b.astype(dtype)).cuda()
        if col_major:
            x = x.t().contiguous().t()
        for _ in range(2):
            assert relerr(s.solve(x).cpu().numpy(), ref) <= tol
            assert relerr(s.solve_adjoint(x)[0].cpu().numpy(), tref) <= tol
        if dtype == np.float64:
            assert relerr(s.solve_refine(x)[0].cpu().numpy(), ref) <= 1e-10
        s.close()


def test_batch_in_blocked_order(cuda, oracle_port):
    from sptrsv_gb300 import SyncFreeSolver
    ms = [_matrix(k, n, low) for k, n, low in (("mesh", 30, True), ("chain", 333, False), ("lists4", 1000, False))]
    s = SyncFreeSolver(batch=[(m.col_ptr, m.row_idx, m.n, m.substitution) for m in ms],
                       values=np.concatenate([m.val for m in ms]), **_blocked(200))
    b = [np.random.default_rng(i).standard_normal(m.n) for i, m in enumerate(ms)]
    x = s.solve(cuda.from_numpy(np.concatenate(b)).cuda()).cpu().numpy()
    at = 0
    for m, bi in zip(ms, b):
        ref = oracle_port.solve(m.col_ptr, m.row_idx, m.val, m.n, m.substitution, bi)
        assert relerr(x[at:at + m.n], ref) <= 1e-12
        at += m.n
    x = s.solve_adjoint(cuda.from_numpy(np.concatenate(b)).cuda())[0].cpu().numpy()
    at = 0
    for m, bi in zip(ms, b):
        t = m.transpose()
        ref = oracle_port.solve(t.col_ptr, t.row_idx, t.val, m.n, t.substitution, bi)
        assert relerr(x[at:at + m.n], ref) <= 1e-12
        at += m.n
    s.close()


def test_infinities_nan_and_signed_zeros_as_the_importer_executor(cuda):
    from sptrsv_gb300 import SyncFreeSolver
    m = _matrix("mesh", 80, True)
    b = np.random.default_rng(5).standard_normal(m.n)
    b[7], b[500] = np.inf, -np.inf
    b.view(np.uint64)[1200] = 0xFFFFFFFFFFFFFFFF
    z = np.full(m.n, -0.0)
    out = []
    for kw in (dict(wsync_batch=1), dict()):
        s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val, **_blocked(320), **kw)
        out.append([s.solve(cuda.from_numpy(v).cuda()).cpu().numpy() for v in (b, z)])
        s.close()
    (u, uz), (v, vz) = out
    assert np.array_equal(np.isnan(u), np.isnan(v)) and np.array_equal(np.isinf(u), np.isinf(v))
    ok = np.isfinite(u)
    assert relerr(v[ok], u[ok]) <= 1e-12
    assert np.array_equal(uz, vz) and np.array_equal(np.signbit(uz), np.signbit(vz))
