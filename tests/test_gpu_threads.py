"""Separate handles used from separate host threads are independent: systems whose walks
ask for very different amounts of shared memory, solved side by side on two streams."""
from __future__ import annotations

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _systems(kind):
    from sptrsv_gb300 import matgen
    if kind == "blocked":   # units of 96 and of 20,000 positions
        m = matgen.laplace2d_lower(150)
        kw = dict(schedule=2, staged=False, warp_sync=True, block=128, ctas_per_sm=0, backoff_ns=0, split=0)
        return [(m, dict(order_block=b, chunk=b, **kw)) for b in (96, 20_000)]
    ms = [matgen.poisson_band(4000, 2.0, 2000, seed=1), matgen.poisson_band(4000, 40.0, 2000, seed=2)]
    return [(m, dict(cluster=0, order_block=2**31 - 1)) for m in ms]


@pytest.mark.parametrize("kind, rhs, call", [("lists", 1, "solve"), ("lists", 1, "adjoint"), ("lists", 2, "solve"),
                                             ("lists", 1, "refine"), ("blocked", 1, "solve")])
def test_two_handles_in_two_threads(cuda, oracle_port, kind, rhs, call):
    from sptrsv_gb300 import SyncFreeSolver
    work = []
    for m, kw in _systems(kind):
        stream = cuda.cuda.Stream()
        with cuda.cuda.stream(stream):
            b = np.random.default_rng(rhs).standard_normal((m.n, rhs))
            t = m.transpose() if call == "adjoint" else m
            ref = oracle_port.solve(t.col_ptr, t.row_idx, t.val, m.n, t.substitution, b).reshape(m.n, rhs)
            s = SyncFreeSolver(m.col_ptr, m.row_idx, m.n, m.substitution, values=m.val, stream=stream, **kw)
            work.append((s, cuda.from_numpy(b).cuda(), cuda.from_numpy(ref).cuda(), stream))
    cuda.cuda.synchronize()
    failures = []

    def run(s, b, ref, stream):
        try:
            with cuda.cuda.stream(stream):
                for _ in range(1500):
                    x = {"solve": lambda: s.solve(b), "adjoint": lambda: s.solve_adjoint(b)[0],
                         "refine": lambda: s.solve_refine(b)[0]}[call]()
                assert float((x - ref).abs().max() / ref.abs().max()) <= (1e-10 if call == "refine" else 1e-12)
        except Exception as e:   # noqa: BLE001 - reported by the main thread
            failures.append(repr(e))

    threads = [threading.Thread(target=run, args=w) for w in work]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not failures, failures
