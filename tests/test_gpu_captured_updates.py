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


class _System:
    """A handle on a stream of its own, its right-hand side, and the oracle's answers."""

    def __init__(self, cuda, oracle, m, dtype, **kw):
        from sptrsv_gb300 import SyncFreeSolver
        self.cuda, self.oracle, self.m = cuda, oracle, m
        self.b = np.random.default_rng(m.n).standard_normal(m.n)
        self.bd = cuda.from_numpy(self.b).cuda()
        self.bf = self.bd.float()
        self.values = cuda.from_numpy(m.val.astype(dtype)).cuda()
        self.s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, sync_check=False,
                                stream=cuda.cuda.current_stream(), order_block=2**31 - 1, **kw)
        self.x = cuda.empty_like(self.bd if dtype == np.float64 else self.bf)

    def update(self):
        b = self.bd if self.x.dtype == self.cuda.float64 else self.bf
        self.s.solve(b, values=self.values, out=self.x)

    def capture(self):
        g = self.cuda.cuda.CUDAGraph()
        with self.cuda.cuda.graph(g, stream=self.cuda.cuda.current_stream()):
            self.update()
        return g

    def check(self, val, names):
        from sptrsv_gb300 import _lib
        m, s = self.m, self.s
        ref = self.oracle.solve(m.col_ptr, m.row_idx, val, m.n, m.substitution, self.b)
        t = type(m)(m.n, m.col_ptr, m.row_idx, val, m.lower).transpose()
        tref = self.oracle.solve(t.col_ptr, t.row_idx, t.val, m.n, t.substitution, self.b)

        def with_option(option, value, call):
            old = s.get_option(option)
            s.set_option(option, value)
            x = call()
            s.set_option(option, old)
            return x

        calls = {"solve": (lambda: s.solve(self.bd), ref, 1e-12),
                 "adjoint": (lambda: s.solve_adjoint(self.bd)[0], tref, 1e-12),
                 "exact": (lambda: with_option(_lib.OPTION_EXACT, 1, lambda: s.solve(self.bd)), ref, 1e-12),
                 "push": (lambda: with_option(_lib.OPTION_SCHEDULE, 1, lambda: s.solve(self.bd)), ref, 1e-12),
                 "exact adjoint": (lambda: with_option(_lib.OPTION_EXACT, 1, lambda: s.solve_adjoint(self.bd)[0]), tref,
                                   1e-12),
                 "refine": (lambda: s.solve_refine(self.bd)[0], ref, 1e-10),
                 "two steps": (lambda: s.solve_refine(self.bd, tol=0.0, max_iter=2)[0], ref, 1e-10),
                 "solve f32": (lambda: s.solve(self.bf), ref, 1e-5),
                 "adjoint f32": (lambda: s.solve_adjoint(self.bf)[0], tref, 1e-5)}
        for name in names:
            call, r, tol = calls[name]
            assert relerr(call().cpu().numpy(), r) <= tol, name


F64 = ("solve", "adjoint", "exact", "exact adjoint", "push", "refine", "two steps", "solve f32", "adjoint f32")
F32 = ("solve f32", "adjoint f32")


@pytest.mark.parametrize("names", [F64, F64[::-1], ("adjoint",), ("solve f32",), ("exact adjoint",), ("refine",), ("two steps",)])
@pytest.mark.parametrize("n, lower", [(33, True), (3000, False)])
def test_replayed_update_reaches_every_form(cuda, oracle_port, own_stream, n, lower, names):
    m = _band(n, lower)
    rng = np.random.default_rng(n)
    sy = _System(cuda, oracle_port, m, np.float64)
    sy.update()
    g = sy.capture()
    sy.check(m.val, names)   # captured, not replayed: the values are still the first ones
    for step in range(3):
        val = m.val * rng.uniform(0.9, 1.1, m.nnz)
        if step == 1:        # an update outside the graph between two replays
            sy.s.set_values(val)
        else:
            sy.values.copy_(cuda.from_numpy(val))
            g.replay()
        sy.check(val, names)
    sy.s.check()


def test_updates_captured_before_and_after_a_form_was_staged(cuda, oracle_port, own_stream):
    """Two graphs, one captured before the transposed weights existed: replayed by turns."""
    m = _band(2000)
    rng = np.random.default_rng(2)
    sy = _System(cuda, oracle_port, m, np.float64)
    sy.update()
    early = sy.capture()
    sy.check(m.val, F64)
    late = sy.capture()
    for g in (late, early, late, late, early):
        val = m.val * rng.uniform(0.9, 1.1, m.nnz)
        sy.values.copy_(cuda.from_numpy(val))
        g.replay()
        sy.check(val, F64)
    sy.s.check()


def test_replayed_update_in_single_precision(cuda, oracle_port, own_stream):
    """FP32 values from a graph, FP64 values set outside it, and FP32 again."""
    m = _band(2500)
    rng = np.random.default_rng(3)
    sy = _System(cuda, oracle_port, m, np.float32)
    sy.update()
    g = sy.capture()
    for step in range(4):
        val = (m.val * rng.uniform(0.9, 1.1, m.nnz)).astype(np.float32)
        if step == 2:
            wide = m.val * rng.uniform(0.9, 1.1, m.nnz)
            sy.s.set_values(wide)
            sy.check(wide, F64)
        sy.values.copy_(cuda.from_numpy(val))
        g.replay()
        sy.check(val.astype(np.float64), F32)
    sy.s.check()


def test_single_precision_update_first_seen_by_a_capture(cuda, oracle_port, own_stream):
    """FP32 values that only a graph ever sets, after FP64 ones: before its first replay the
    FP64 values count, then the graph's, then whichever came last."""
    m = _band(1500)
    rng = np.random.default_rng(4)
    sy = _System(cuda, oracle_port, m, np.float64)
    sy.update()
    sy.values, sy.x = sy.values.float(), sy.x.float()
    g = sy.capture()
    sy.check(m.val, F32)
    for step in range(3):
        val = (m.val * rng.uniform(0.9, 1.1, m.nnz)).astype(np.float32)
        sy.values.copy_(cuda.from_numpy(val))
        g.replay()
        sy.check(val.astype(np.float64), F32)
        wide = m.val * rng.uniform(0.9, 1.1, m.nnz)
        sy.s.set_values(wide)
        sy.check(wide, F32 if step % 2 else F64)
        if step == 2:   # an FP64 solve of the values set last, although an FP32 replay came between
            g.replay()
            sy.check(wide, ("adjoint", "exact"))
    sy.s.check()


@pytest.mark.parametrize("rhs, steps", [(1, 1), (1, 2), (8, 1)])
def test_refinement_graph_follows_new_values(cuda, oracle_port, rhs, steps):
    from sptrsv_gb300 import SyncFreeSolver
    m = _band(4000)
    rng = np.random.default_rng(rhs)
    b = rng.standard_normal((m.n, rhs))
    s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val)
    bd = cuda.from_numpy(b).cuda()
    x = cuda.empty_like(bd)
    g = s.graph(bd, x, kind=1, count=steps)
    for _ in range(2):
        val = m.val * rng.uniform(0.9, 1.1, m.nnz)
        s.set_values(val)
        g.replay()
        s.check()
        ref = oracle_port.solve(m.col_ptr, m.row_idx, val, m.n, m.substitution, b)
        assert relerr(x.cpu().numpy(), ref) <= 1e-10
    g.close()


@pytest.mark.parametrize("case", ["adjoint", "single precision block", "refined block"])
def test_tables_first_needed_inside_a_capture(cuda, oracle_port, own_stream, case):
    """A blocked layout's tables are built outside captures; a walk captured before they
    exist takes an executor that does without them."""
    from sptrsv_gb300 import SyncFreeSolver, matgen
    stream = cuda.cuda.current_stream()
    if case == "adjoint":    # rows of more than four entries, columns of at most four
        m = matgen.banded_random_lower(3000, np.random.default_rng(1).integers(0, 5, 3000), 60, 7)
        kw = dict(schedule=2, staged=False, warp_sync=True, order_block=300, chunk=300, block=128, ctas_per_sm=0,
                  backoff_ns=0, split=0)
    else:
        m, kw = matgen.laplace2d_lower(150), {}
    s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val, sync_check=False, stream=stream, **kw)

    def block(rhs, dtype):
        return cuda.from_numpy(np.random.default_rng(rhs).standard_normal((m.n, rhs)).astype(dtype)).cuda()

    b = block(*{"adjoint": (1, np.float64), "single precision block": (14, np.float32),
                "refined block": (16, np.float64)}[case])
    x = cuda.empty_like(b)
    if case == "adjoint":
        s.solve(b)
        call = lambda: s.solve_adjoint(b, out=x)   # noqa: E731
    elif case == "single precision block":
        s.solve(block(7, np.float64))              # the value words reach for 14 in FP32
        s.solve(block(1, np.float32))
        call = lambda: s.solve(b, out=x)           # noqa: E731
    else:                                          # workspaces and forms from the FP64 residual's step
        from sptrsv_gb300 import _lib
        s.set_option(_lib.OPTION_FUSED_REFINE, 1)
        s.solve_refine(b)
        s.set_option(_lib.OPTION_FUSED_REFINE, 2)
        call = lambda: s.solve_refine(b, out=x, tol=0.0, max_iter=1)   # noqa: E731
    stream.synchronize()
    g = cuda.cuda.CUDAGraph()
    with cuda.cuda.graph(g, stream=stream):
        call()
    t = m.transpose() if case == "adjoint" else m
    ref = oracle_port.solve(t.col_ptr, t.row_idx, t.val, m.n, t.substitution, b.double().cpu().numpy())
    for _ in range(2):
        x.zero_()
        g.replay()
        assert relerr(x.cpu().numpy(), ref) <= {"adjoint": 1e-12, "single precision block": 1e-5,
                                                "refined block": 1e-10}[case]
        call()    # the tables are there from now on
    s.check()
