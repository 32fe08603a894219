"""One-cluster executor (SPTRSV_OPTION_CLUSTER): sizes around its tiles (32 unknowns
per warp, runs of 32 / 128 / 256 walk indices, 16 CTAs), lists longer than a warp's
buffer, systems past its shared memory, and values that must not be mistaken for an
unpublished word. FP64 <= 1e-12 relative against the oracle (max norm, the tolerance
of every pull executor), FP32 <= 1e-5."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def relerr(x, ref):
    x, ref = np.asarray(x, np.float64).ravel(), np.asarray(ref, np.float64).ravel()
    return float(np.max(np.abs(x - ref)) / max(np.max(np.abs(ref)), 1e-300))


def _matrix(kind, n, lower):
    from sptrsv_gb300 import matgen
    if kind == "band":
        return matgen.poisson_band(n, 6.0, max(n // 4, 2), seed=n, lower=lower)
    if kind == "thin":       # a few unknowns per level: runs of 256
        return matgen.poisson_band(n, 6.0, 40, seed=n, lower=lower)
    if kind == "deep":       # more than 1,000 dependencies per level: runs of 32
        return matgen.poisson_band(n, 14.0, n // 2, seed=n, lower=lower)
    if kind == "star":       # transposed: one list of n - 1 entries
        return matgen.star(n, lower=lower)
    return matgen.dense_lower(n, lower=lower)


@pytest.mark.parametrize("lower", [True, False])
@pytest.mark.parametrize("kind, n", [("band", 1), ("band", 2), ("band", 31), ("band", 33), ("band", 511),
                                     ("band", 513), ("band", 2047), ("band", 2049), ("thin", 4095), ("thin", 4097),
                                     ("thin", 20_001), ("deep", 30_001), ("star", 3000), ("dense", 300)])
def test_cluster_solves_match_the_oracle(cuda, oracle_port, kind, n, lower):
    from sptrsv_gb300 import SyncFreeSolver
    m = _matrix(kind, n, lower)
    rng = np.random.default_rng(n)
    b, g = rng.standard_normal(n), rng.standard_normal(n)
    ref = oracle_port.solve(m.col_ptr, m.row_idx, m.val, n, m.substitution, b)
    t = m.transpose()
    tref = oracle_port.solve(t.col_ptr, t.row_idx, t.val, n, t.substitution, g)
    for dtype, tol in ((np.float64, 1e-12), (np.float32, 1e-5)):
        s = SyncFreeSolver(m.col_ptr, m.row_idx, n, m.substitution, values=m.val.astype(dtype), cluster=1)
        bd, gd = cuda.from_numpy(b.astype(dtype)).cuda(), cuda.from_numpy(g.astype(dtype)).cuda()
        for view in (bd, bd.reshape(-1, 1)):
            assert relerr(s.solve(view).cpu().numpy(), ref) <= tol
        lam, _ = s.solve_adjoint(gd)
        assert relerr(lam.cpu().numpy(), tref) <= tol
        s.close()


def test_cluster_falls_back_where_the_values_do_not_fit(cuda, oracle_port):
    """500,001 FP64 values exceed 16 CTAs' shared memory: the general executor runs."""
    from sptrsv_gb300 import SyncFreeSolver, matgen
    m = matgen.poisson_band(500_001, 2.0, 200_000, seed=3)
    b = np.random.default_rng(3).standard_normal(m.n)
    s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val, cluster=1)
    ref = oracle_port.solve(m.col_ptr, m.row_idx, m.val, m.n, m.substitution, b)
    assert relerr(s.solve(cuda.from_numpy(b).cuda()).cpu().numpy(), ref) <= 1e-12


def test_cluster_keeps_infinities_and_nan(cuda):
    """Infinities and NaN (the all-ones pattern of an unpublished word among them) reach
    the same unknowns as in the general executor."""
    from sptrsv_gb300 import SyncFreeSolver
    m = _matrix("band", 3001, True)
    b = np.random.default_rng(5).standard_normal(m.n)
    b[7], b[500] = np.inf, -np.inf
    b.view(np.uint64)[1200] = 0xFFFFFFFFFFFFFFFF
    out = []
    for mode in (0, 1):
        s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val, cluster=mode)
        out.append(s.solve(cuda.from_numpy(b).cuda()).cpu().numpy())
    assert np.array_equal(np.isnan(out[0]), np.isnan(out[1]))
    assert np.array_equal(np.isinf(out[0]), np.isinf(out[1]))
    ok = np.isfinite(out[0])
    assert relerr(out[1][ok], out[0][ok]) <= 1e-12


def test_cluster_option_values(cuda):
    from sptrsv_gb300 import SptrsvError, SyncFreeSolver, _lib
    m = _matrix("band", 100, True)
    s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val)
    assert s.get_option(_lib.OPTION_CLUSTER) == 2
    for v in (0, 1, 2):
        s.set_option(_lib.OPTION_CLUSTER, v)
        assert s.get_option(_lib.OPTION_CLUSTER) == v
    for v in (-1, 3):
        with pytest.raises(SptrsvError):
            s.set_option(_lib.OPTION_CLUSTER, v)
