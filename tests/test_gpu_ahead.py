"""Level-order executor with lists staged ahead: sizes around its segments (32 walk
indices) and CTAs (8 segments), lists longer than a warp's buffer (640 entries), chains
inside a segment, and both precisions and directions. FP64 <= 1e-12 relative against the
oracle (max norm, the tolerance of every pull executor), FP32 <= 1e-5. cluster=0 keeps
the one-cluster executor off these small systems."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def relerr(x, ref):
    x, ref = np.asarray(x, np.float64).ravel(), np.asarray(ref, np.float64).ravel()
    return float(np.max(np.abs(x - ref)) / max(np.max(np.abs(ref)), 1e-300))


def _matrix(kind, n, lower):
    from sptrsv_gb300 import matgen
    return {"band": lambda: matgen.poisson_band(n, 7.0, max(n // 3, 2), seed=n, lower=lower),
            "chain": lambda: matgen.chain(n, lower=lower), "diagonal": lambda: matgen.diagonal(n, lower=lower),
            "dense": lambda: matgen.dense_lower(n, lower=lower), "mesh": lambda: matgen.laplace2d_lower(n, lower=lower),
            "power": lambda: matgen.power_law_band(n, 9 * n, n // 2, seed=n, kmax=30, lower=lower)}[kind]()


# the automatic plan, and the explicit settings that ask for the same walk
@pytest.mark.parametrize("kw", [dict(), dict(schedule=2, staged=False, warp_sync=True, ctas_per_sm=1, wsync_batch=1,
                                             chunk=256, block=256, backoff_ns=0, split=0)])
@pytest.mark.parametrize("lower", [True, False])
@pytest.mark.parametrize("kind, n", [("band", 1), ("band", 31), ("band", 33), ("band", 255), ("band", 257),
                                     ("band", 40_001), ("chain", 700), ("diagonal", 5000), ("dense", 700),
                                     ("mesh", 40), ("power", 20_000)])
def test_staged_ahead_solves_match_the_oracle(cuda, oracle_port, kind, n, lower, kw):
    from sptrsv_gb300 import SyncFreeSolver
    m = _matrix(kind, n, lower)
    rng = np.random.default_rng(n)
    b, g = rng.standard_normal(m.n), rng.standard_normal(m.n)
    ref = oracle_port.solve(m.col_ptr, m.row_idx, m.val, m.n, m.substitution, b)
    t = m.transpose()
    tref = oracle_port.solve(t.col_ptr, t.row_idx, t.val, m.n, t.substitution, g)
    for dtype, tol in ((np.float64, 1e-12), (np.float32, 1e-5)):
        s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val.astype(dtype), cluster=0,
                           order_block=2**31 - 1, **kw)
        for _ in range(2):   # the ticket starts over
            x = s.solve(cuda.from_numpy(b.astype(dtype)).cuda())
            assert relerr(x.cpu().numpy(), ref) <= tol
            lam, _ = s.solve_adjoint(cuda.from_numpy(g.astype(dtype)).cuda())
            assert relerr(lam.cpu().numpy(), tref) <= tol
        s.close()


@pytest.mark.parametrize("lower", [True, False])
@pytest.mark.parametrize("kind, n", [("star", 40), ("star", 70), ("star", 3000), ("power", 2000), ("power", 20_000),
                                     ("few", 1025), ("few", 5000)])
def test_split_lists_match_the_oracle(cuda, oracle_port, kind, n, lower):
    """Lists of up to 3,000 entries over 2 to 32 lanes, whole and partial segments, packing blocks of 1,024."""
    from sptrsv_gb300 import SyncFreeSolver, matgen
    if kind == "star":
        m = matgen.star(n, lower=lower)
    elif kind == "power":
        m = matgen.power_law_band(n, 9 * n, n // 4, seed=n, lower=lower)
    else:   # a few long columns among columns of two entries
        counts = np.where(np.arange(n) % 97 == 0, 200, 2)
        m = matgen.banded_random_lower(n, counts, n // 2, n, lower=lower)
    s64 = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val, cluster=0)
    if not lower:
        assert s64.info()["split"] == 32
    s64.close()
    rng = np.random.default_rng(n)
    b = rng.standard_normal(m.n)
    ref = oracle_port.solve(m.col_ptr, m.row_idx, m.val, m.n, m.substitution, b)
    t = m.transpose()
    tref = oracle_port.solve(t.col_ptr, t.row_idx, t.val, m.n, t.substitution, b)
    for dtype, tol in ((np.float64, 1e-12), (np.float32, 1e-5)):
        s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val.astype(dtype), cluster=0)
        bd = cuda.from_numpy(b.astype(dtype)).cuda()
        for _ in range(2):
            assert relerr(s.solve(bd).cpu().numpy(), ref) <= tol
            assert relerr(s.solve_adjoint(bd)[0].cpu().numpy(), tref) <= tol
        s.close()


def test_infinities_and_nan_reach_the_same_unknowns(cuda):
    """Against the executor that reads its lists from global memory (128 threads per CTA)."""
    from sptrsv_gb300 import SyncFreeSolver
    m = _matrix("band", 3001, True)
    b = np.random.default_rng(5).standard_normal(m.n)
    b[7], b[500] = np.inf, -np.inf
    b.view(np.uint64)[1200] = 0xFFFFFFFFFFFFFFFF
    out = []
    for kw in (dict(block=128), dict()):
        s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val, cluster=0, **kw)
        out.append(s.solve(cuda.from_numpy(b).cuda()).cpu().numpy())
    assert np.array_equal(np.isnan(out[0]), np.isnan(out[1]))
    assert np.array_equal(np.isinf(out[0]), np.isinf(out[1]))
    ok = np.isfinite(out[0])
    assert relerr(out[1][ok], out[0][ok]) <= 1e-12


@pytest.mark.parametrize("chunk, split", [(32, 4), (33, 4), (100, 8), (256, 8), (256, 32), (1000, 5)])
@pytest.mark.parametrize("kind, n", [("star", 33), ("star", 700), ("few", 1025), ("power", 5003), ("chain", 300)])
def test_pieces_of_split_lists(cuda, oracle_port, kind, n, chunk, split):
    """Pieces packed on the device for the executor that splits lists in chunks: ranges and segments of every fill,
    chunks cut at their segment limit, both directions (the transposed walk starts with a partial chunk)."""
    from sptrsv_gb300 import SyncFreeSolver, matgen
    m = {"star": lambda: matgen.star(n, lower=False), "chain": lambda: matgen.chain(n, lower=False),
         "power": lambda: matgen.power_law_band(n, 9 * n, n // 4, seed=n, lower=False),
         "few": lambda: matgen.banded_random_lower(n, np.where(np.arange(n) % 97 == 0, 200, 2), n // 2, n,
                                                   lower=False)}[kind]()
    b = np.random.default_rng(n).standard_normal(m.n)
    ref = oracle_port.solve(m.col_ptr, m.row_idx, m.val, m.n, m.substitution, b)
    t = m.transpose()
    tref = oracle_port.solve(t.col_ptr, t.row_idx, t.val, m.n, t.substitution, b)
    s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val, schedule=2, staged=False,
                       warp_sync=True, order_block=2**31 - 1, chunk=chunk, split=split, wsync_batch=2, cluster=0)
    bd = cuda.from_numpy(b).cuda()
    for _ in range(2):
        assert relerr(s.solve(bd).cpu().numpy(), ref) <= 1e-12
        assert relerr(s.solve_adjoint(bd)[0].cpu().numpy(), tref) <= 1e-12
    s.close()
