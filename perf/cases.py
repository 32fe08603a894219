"""The solver's working range as timed cases.

Each case is one call pattern of a program that uses this package, at sizes of
the repository's own workloads: the 10,000-row system, the 1414 x 1414 mesh
triangle, the power-law triangles, the 1M-row band system at 1-64 right-hand
sides, batches of uneven systems, refinement, differentiable solves, value
updates, new patterns and the drop-in host call.

Matrices are drawn on the GPU from the seed alone, in the package's storage
(CSC, 0-based int32, rows ascending, the diagonal first in a lower column and
last in an upper one), strictly diagonally dominant by rows and by columns.
``exact`` solves the same systems by the fixed point x = D^-1 (b - N x) in
64-bit torch, which converges to rounding for such matrices.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parents[1] / "benchmark-sptrsv_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import sptrsv_gb300 as sp  # noqa: E402


# ------------------------------------------------------------------ cases

def listed():
    return [
        # one right-hand side of the smallest member of a batch: a call's fixed cost
        {"name": "solve_1k", "call": "solve", "shape": "band", "n": 1000, "mean": 8.0, "band": 400, "lower": True,
         "rhs": 1, "dtype": "f64", "col_major": False},
        # the 10,000-row system: a small factor applied inside an outer iteration
        {"name": "solve_10k", "call": "solve", "shape": "band", "n": 10_000, "mean": 8.0, "band": 2000,
         "lower": True, "rhs": 1, "dtype": "f64", "col_major": False},
        # the mesh triangle, applied as a preconditioner (asynchronous calls)
        {"name": "solve_mesh_2m", "call": "solve_async", "shape": "mesh", "n": 1414 * 1414, "mean": 2.0,
         "band": 1414, "lower": True, "rhs": 1, "dtype": "f64", "col_major": False},
        # the power-law upper triangle, backward substitution: rows of up to ~1,000 entries
        {"name": "solve_powerlaw_bwd_4m", "call": "solve", "shape": "power", "n": 4_194_304, "mean": 8.0,
         "band": 50_000, "lower": False, "rhs": 1, "dtype": "f64", "col_major": False},
        # a power-law lower triangle in single precision, odd size
        {"name": "solve_powerlaw_f32_1m", "call": "solve", "shape": "power", "n": 1_048_577, "mean": 8.0,
         "band": 50_000, "lower": True, "rhs": 1, "dtype": "f32", "col_major": False},
        # a deep, narrow band factor: thousands of small level sets
        {"name": "solve_deep_150k", "call": "solve", "shape": "band", "n": 150_001, "mean": 6.0, "band": 200,
         "lower": False, "rhs": 1, "dtype": "f64", "col_major": False},
        # a block of 64 right-hand sides, stored column by column
        {"name": "solve_band_1m_rhs64", "call": "solve", "shape": "band", "n": 1_000_000, "mean": 9.0,
         "band": 20_000, "lower": True, "rhs": 64, "dtype": "f64", "col_major": True},
        # single-precision solve refined to double accuracy
        {"name": "refine_band_1m_rhs16", "call": "refine", "shape": "band", "n": 1_000_000, "mean": 9.0,
         "band": 20_000, "lower": True, "rhs": 16, "dtype": "f64", "col_major": True},
        # independent uneven systems in one launch, lower and upper by turns
        {"name": "batch_64", "call": "batch", "shape": "uneven", "n": 200_000, "count": 64, "rhs": 4},
        # a training step: new values, differentiable solve, gradients of values and right-hand sides
        {"name": "train_band_500k_rhs8", "call": "train", "shape": "band", "n": 500_000, "mean": 9.0,
         "band": 20_000, "lower": True, "rhs": 8, "dtype": "f64", "col_major": False},
        # a time step: the same pattern with new values, one solve
        {"name": "update_mesh_1m", "call": "update", "shape": "mesh", "n": 1000 * 1000, "mean": 2.0, "band": 1000,
         "lower": True, "rhs": 1, "dtype": "f64", "col_major": False},
        # a new pattern: analysis, values, one solve through the drop-in host call
        {"name": "drop_in_300k", "call": "drop_in", "shape": "band", "n": 300_000, "mean": 9.0, "band": 20_000,
         "lower": True, "rhs": 1, "dtype": "f64", "col_major": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["solve", "solve", "solve", "solve_async", "refine", "batch", "train", "update", "drop_in"])
    if call == "batch":
        return {"call": call, "shape": "uneven", "n": _log_int(rng, 4_000, 200_000), "count": rng.randint(8, 64),
                "rhs": rng.randint(1, 4)}
    shape = rng.choice(["band", "band", "mesh", "power"])
    top = {"solve": 4_000_000, "solve_async": 4_000_000, "refine": 1_000_000, "train": 500_000,
           "update": 1_000_000, "drop_in": 300_000}[call]
    n = _log_int(rng, 1_000, min(top, {"band": 1_000_000, "mesh": 2_000_000, "power": 4_000_000}[shape]))
    rhs = {"solve": rng.choice([1, 1, 1, 2, 4, 8, 16, 33, 64]), "refine": rng.choice([1, 1, 4, 16, 31]),
           "train": rng.choice([1, 4, 8])}.get(call, 1)
    if rhs > 1:
        n = min(n, 64_000_000 // rhs // (1 if shape == "band" else 4), 1_000_000)
    case = {"call": call, "shape": shape, "n": n, "lower": rng.random() < 0.6, "rhs": rhs,
            "dtype": "f32" if call in ("solve", "solve_async") and rng.random() < 0.25 else "f64",
            "col_major": rhs > 1 and call in ("solve", "refine") and rng.random() < 0.5}
    if shape == "mesh":
        g = max(int(math.isqrt(n)), 8)
        case.update(n=g * g, mean=2.0, band=g)
    elif shape == "power":
        case.update(mean=8.0, band=min(50_000, max(n // 4, 64)))
    else:
        # bands of n/50 to n/2 rows, at most 20,000 (level sets a few hundred wide at the larger sizes)
        case.update(mean=float(rng.randint(2, 12)),
                    band=min(20_000, max(int(n * math.exp(rng.uniform(math.log(0.02), math.log(0.5)))), 64)))
    return case


# ------------------------------------------------------------------ matrices

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _power_scale(mean, kmax=1000, alpha=2.1):
    """The factor that makes clip(round(factor * k), 1, kmax), k ~ k^-alpha, average ``mean``."""
    k = np.arange(1, kmax + 1, dtype=np.float64)
    pmf = k ** -alpha
    pmf /= pmf.sum()
    f = mean / float((pmf * k).sum())
    for _ in range(8):
        f *= mean / float((pmf * np.clip(np.rint(k * f), 1, kmax)).sum())
    return np.cumsum(pmf), f


def _off_diagonals(shape, n, mean, band, g):
    """(column, row) of the entries below the diagonal, sorted by column then row."""
    j = torch.arange(n, device="cuda", dtype=torch.int64)
    if shape == "mesh":
        right = j[(j % band) < band - 1]
        down = j[j < n - band]
        key = torch.cat([right * n + right + 1, down * n + down + band]).sort().values
    else:
        if shape == "power":
            cdf, f = _power_scale(mean)
            u = torch.rand(n, device="cuda", dtype=torch.float64, generator=g)
            k = torch.searchsorted(torch.from_numpy(cdf).cuda(), u, right=True) + 1
            k = (k.clamp_(max=1000) * f).round().clamp_(1, 1000).long()
        else:
            k = torch.poisson(torch.full((n,), float(mean), device="cuda", dtype=torch.float32), generator=g).long()
        room = (torch.clamp(j + band, max=n) - (j + 1)).clamp_(min=0)
        col = torch.repeat_interleave(j, torch.minimum(k, room))
        span = room[col]
        u = torch.rand(col.numel(), device="cuda", dtype=torch.float64, generator=g)
        row = col + 1 + torch.minimum((u * span).long(), span - 1)
        key = torch.unique(col * n + row)
    return key // n, key % n


def _triangle(shape, n, mean, band, lower, g):
    """(column pointers, row indices, column of every entry, diagonal positions) on the GPU."""
    col, row = _off_diagonals(shape, n, mean, band, g)
    if not lower:
        key = (row * n + col).sort().values
        col, row = key // n, key % n
    d = torch.arange(n, device="cuda", dtype=torch.int64)
    count = torch.bincount(col, minlength=n) + 1
    ptr = torch.zeros(n + 1, device="cuda", dtype=torch.int64)
    torch.cumsum(count, 0, out=ptr[1:])
    at = torch.arange(col.numel(), device="cuda") + col + (1 if lower else 0)
    diag = ptr[:-1] if lower else ptr[1:] - 1
    rows = torch.empty(col.numel() + n, device="cuda", dtype=torch.int32)
    cols = torch.empty_like(rows)
    rows[at], cols[at] = row.int(), col.int()
    rows[diag], cols[diag] = d.int(), d.int()
    return ptr.int(), rows, cols, diag


def _values(shape, rows, cols, diag, g):
    """Off-diagonals in [-0.1, 0.1] and a dominant diagonal; the mesh has -1 (a little off) and 4."""
    n, nnz = diag.numel(), rows.numel()
    u = torch.rand(nnz, device="cuda", dtype=torch.float64, generator=g)
    if shape == "mesh":
        val = u.mul_(0.05).sub_(1.0)
        val[diag] += 5.0
        return val
    val = u.mul_(0.2).sub_(0.1)
    size = torch.bincount(rows, minlength=n) + torch.bincount(cols, minlength=n) - 2
    val[diag] = 1.0 + torch.rand(n, device="cuda", dtype=torch.float64, generator=g) + 0.1 * size
    return val


def _right_hand_sides(n, rhs, col_major, g):
    if col_major:
        return torch.randn(rhs, n, device="cuda", dtype=torch.float64, generator=g).t()
    return torch.randn(n, rhs, device="cuda", dtype=torch.float64, generator=g)


def _system(case, seed):
    g = _generator(seed)
    # a training program keeps its pattern: there the seed draws values and vectors only
    pattern = _generator(case["n"]) if case["call"] == "train" else g
    ptr, rows, cols, diag = _triangle(case["shape"], case["n"], case["mean"], case["band"], case["lower"], pattern)
    val = _values(case["shape"], rows, cols, diag, g)
    b = _right_hand_sides(case["n"], case["rhs"], case["col_major"], g)
    if case["rhs"] == 1:
        b = b.reshape(-1)
    if case["dtype"] == "f32":
        val, b = val.float(), b.float()
    return ptr, rows, cols, diag, val, b, g


def _batch(case, seed):
    """Uneven members: sizes spread over the logarithm from 1,000 to n, 3-20 entries a column, bands of
    100-10,000 rows."""
    r = np.random.default_rng(seed)
    g = _generator(seed)
    out = []
    for s in range(case["count"]):
        n = int(1000 * (case["n"] / 1000) ** (s * 0.6180339887498949 % 1.0))
        mean, band = float(r.integers(2, 20)), int(r.integers(100, 10_001))
        ptr, rows, cols, diag = _triangle("band", n, mean, band, s % 2 == 0, g)
        out.append((ptr, rows, cols, diag, _values("band", rows, cols, diag, g)))
    total = sum(m[3].numel() for m in out)
    return out, _right_hand_sides(total, case["rhs"], False, g)


# ------------------------------------------------------------------ the calls

def prepare(case, seed):
    call = case["call"]
    if call == "batch":
        members, b = _batch(case, seed)
        solver = sp.SyncFreeSolver(batch=[(m[0].cpu().numpy(), m[1].cpu().numpy(), m[3].numel(), s % 2)
                                          for s, m in enumerate(members)])
        solver.set_values(torch.cat([m[4] for m in members]))
        return {"call": call, "solver": solver, "b": b}
    ptr, rows, _, _, val, b, g = _system(case, seed)
    sub = sp.SUBSTITUTION_FORWARD if case["lower"] else sp.SUBSTITUTION_BACKWARD
    if call == "drop_in":
        n = case["n"]
        return {"call": call, "args": (ptr.cpu().numpy(), rows.cpu().numpy(), val.cpu().numpy(), n, n, rows.numel(),
                                       sub, 1, sp.OPT_WARP_AUTO), "b": b.cpu().numpy(), "x": np.empty(n)}
    if call == "solve_async":
        solver = sp.SyncFreeSolver(ptr, rows, case["n"], sub, values=val, sync_check=False)
    else:
        solver = sp.SyncFreeSolver(ptr, rows, case["n"], sub, values=val)
    state = {"call": call, "solver": solver, "b": b}
    if call == "update":
        state["values"] = val
    if call == "train":
        state["values"] = val.requires_grad_(True)
        state["b"] = b.requires_grad_(True)
        state["gx"] = torch.randn(b.shape, device="cuda", dtype=b.dtype, generator=g)
    return state


def run(state):
    call = state["call"]
    if call in ("solve", "solve_async", "batch"):
        return state["solver"].solve(state["b"])
    if call == "refine":
        return state["solver"].solve_refine(state["b"])[0]
    if call == "update":
        return state["solver"].solve(state["b"], values=state["values"])
    if call == "train":
        x = sp.sparse_triangular_solve(state["solver"], state["values"], state["b"])
        db, dv = torch.autograd.grad(x, (state["b"], state["values"]), state["gx"])
        return x.detach(), db, dv
    # drop-in: host arrays in, x out, one analysis and one solve
    sp.sptrsv_syncfree_cuda(*state["args"], state["x"], state["b"], repeat=1)
    return state["x"]


# ------------------------------------------------------------------ what a pass needs

def work(case):
    if case["call"] == "batch":
        lo, hi = math.log(1000), math.log(case["n"])
        n = case["count"] * (math.exp(hi) - math.exp(lo)) / (hi - lo)
        nnz = n * 11.5
        return {"bytes": nnz * 12 + n * 4 + 2 * n * case["rhs"] * 8, "flops": 2 * nnz * case["rhs"]}
    n, rhs = case["n"], case["rhs"]
    size = 4 if case["dtype"] == "f32" else 8
    nnz = n * (1 + case["mean"])
    solve = nnz * (4 + size) + 4 * n + 2 * n * rhs * size
    flops = 2 * nnz * rhs
    if case["call"] == "train":  # x, lambda and the gradient of every stored value
        return {"bytes": 2 * solve + nnz * size, "flops": 3 * flops}
    return {"bytes": solve, "flops": flops}


# ------------------------------------------------------------------ 64-bit results

def _fixed_point(out_index, in_index, w, diag_val, b):
    """x with diag_val * x + sum over entries of w * x[in_index] (added at out_index) = b."""
    n, rhs = b.shape
    a = torch.sparse_coo_tensor(torch.stack([out_index, in_index]), w, (n, n)).coalesce().to_sparse_csr()
    parts = []
    for k in range(0, rhs, 16):
        bk = b[:, k:k + 16].contiguous()
        x = bk / diag_val[:, None]
        for _ in range(400):
            y = (bk - a @ x) / diag_val[:, None]
            step = (y - x).abs().max() / y.abs().max()
            x = y
            if float(step) < 1e-17:
                break
        parts.append(x)
    return torch.cat(parts, 1)


def _solve64(rows, cols, diag, val, b, transposed=False):
    rows, cols, val, b = rows.long(), cols.long(), val.double(), b.double()
    off = torch.ones(rows.numel(), device=rows.device, dtype=torch.bool)
    off[diag] = False
    r, c = (cols, rows) if transposed else (rows, cols)
    return _fixed_point(r[off], c[off], val[off], val[diag], b.reshape(b.shape[0], -1)).reshape(b.shape)


def exact(case, seed):
    if case["call"] == "batch":
        members, b = _batch(case, seed)
        parts, at = [], 0
        for _, rows, cols, diag, val in members:
            n = diag.numel()
            parts.append(_solve64(rows, cols, diag, val, b[at:at + n]))
            at += n
        return torch.cat(parts)
    _, rows, cols, diag, val, b, g = _system(case, seed)
    x = _solve64(rows, cols, diag, val, b)
    if case["call"] == "drop_in":
        return x.cpu().numpy()
    if case["call"] != "train":
        return x
    gx = torch.randn(b.shape, device="cuda", dtype=b.dtype, generator=g)
    lam = _solve64(rows, cols, diag, val, gx, transposed=True)
    dv = torch.empty_like(val)
    for i in range(0, val.numel(), 1 << 22):
        r, c = rows[i:i + (1 << 22)].long(), cols[i:i + (1 << 22)].long()
        dv[i:i + (1 << 22)] = -(lam[r] * x[c]).reshape(r.numel(), -1).sum(1)
    return x, lam, dv
