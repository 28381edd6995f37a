"""The work this engine is asked to do, as cases that can be timed.

Every case goes through the public Python API (``PdlpSolver``, ``batch_solve``,
``Server``) on host arrays, the way a program that embeds the engine calls it:

* ``solve``     -- an LP that stays loaded is solved (again): root LPs, repeated
  solves of one model, the headline benchmark's step.
* ``e2e``       -- a new solver per pass: load (scaling), solve, read x and y.
* ``dive``      -- a branch-and-bound dive step: one column's bounds change, the
  parent's x and y warm-start the solve.
* ``batch``     -- many independent LPs of uneven sizes in one call.
* ``serve``     -- node LPs of one base LP submitted to a running server and
  waited for.

LPs: random sparse (4-12 nonzeros per column), transportation, and power-law
column lengths -- the generators and shapes of the benchmark and the tests.
Random LPs of the ``solve``, ``e2e`` and ``batch`` cases carry an objective and
right-hand sides built around a known optimal vertex, so that the exact answer
is known.
"""
from __future__ import annotations

import math

import numpy as np

from mipx_b200 import generators as G
from mipx_b200.pdlp import PdlpOptions, PdlpSolver, Precision, Server, batch_solve

CUTS = 50  # most cut rows of a node LP


def listed():
    return [
        # the smallest model a MIP code sends: latency of the iteration loop alone
        {"name": "solve_60x150", "kind": "solve", "lp": "random", "m": 60, "n": 150, "tol": 1e-6, "fp64": False},
        # a small model from arrays to answer, the way a one-off caller uses the library
        {"name": "e2e_400x1000", "kind": "e2e", "lp": "random", "m": 400, "n": 1000, "tol": 1e-6, "fp64": False},
        # the single-LP size of the benchmark
        {"name": "solve_2000x5000", "kind": "solve", "lp": "random", "m": 2000, "n": 5000, "tol": 1e-6, "fp64": False},
        # a dive step on a model of ragged size: rescaling, new device image, warm start
        {"name": "dive_1013x2531", "kind": "dive", "lp": "random", "m": 1013, "n": 2531, "tol": 1e-6, "fp64": False},
        # FP64 throughout on the serving workload's base size
        {"name": "solve_20000x50000_fp64", "kind": "solve", "lp": "random", "m": 20000, "n": 50000, "tol": 1e-4,
         "fp64": True},
        # two entries per column, long rows: supply and demand rows of a small network
        {"name": "transport_97x131", "kind": "solve", "lp": "transport", "m": 97, "n": 131, "tol": 1e-4, "fp64": False},
        # the benchmark's transportation LP, an approximate answer (a start for a heuristic)
        {"name": "transport_1000x1000", "kind": "solve", "lp": "transport", "m": 1000, "n": 1000, "tol": 1e-1,
         "fp64": False},
        # power-law column lengths: the size that just leaves the L2 in FP64
        {"name": "powerlaw_25000x100000", "kind": "solve", "lp": "powerlaw", "m": 25000, "n": 100000, "tol": 1e-3,
         "fp64": False},
        # the headline LP of the benchmark, an approximate answer
        {"name": "powerlaw_500000x2000000", "kind": "solve", "lp": "powerlaw", "m": 500000, "n": 2000000,
         "tol": 1e-2, "fp64": False},
        # a handful of subproblems solved together in FP64
        {"name": "batch_12_fp64", "kind": "batch", "lp": "random", "count": 12, "median": 400, "tol": 1e-5,
         "fp64": True},
        # the batched workload's size distribution
        {"name": "batch_64", "kind": "batch", "lp": "random", "count": 64, "median": 1500, "tol": 1e-5, "fp64": False},
        # node LPs of one base LP through the server
        {"name": "serve_16_of_1000x2500", "kind": "serve", "lp": "random", "m": 1000, "n": 2500, "count": 16,
         "tol": 1e-4, "fp64": False},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["solve", "solve", "solve", "transport", "powerlaw", "e2e", "dive", "batch", "serve"])
    fp64 = rng.random() < 0.3
    if kind == "transport":
        return {"kind": "solve", "lp": "transport", "m": log(20, 300), "n": log(20, 300),
                "tol": rng.choice([1e-2, 1e-3]), "fp64": fp64}
    if kind == "powerlaw":
        m = log(20000, 300000)
        return {"kind": "solve", "lp": "powerlaw", "m": m, "n": int(m * rng.uniform(2.5, 4.0)),
                "tol": rng.choice([1e-1, 1e-2]), "fp64": fp64}
    if kind == "batch":
        return {"kind": "batch", "lp": "random", "count": log(3, 48), "median": log(200, 1500),
                "tol": rng.choice([1e-4, 1e-5]), "fp64": fp64}
    if kind == "serve":
        m = log(200, 1200)
        return {"kind": "serve", "lp": "random", "m": m, "n": int(m * rng.uniform(2.0, 3.0)), "count": log(2, 16),
                "tol": 1e-4, "fp64": False}
    m = log(50, 20000) if kind == "solve" else log(100, 3000)
    return {"kind": kind, "lp": "random", "m": m, "n": int(m * rng.uniform(2.0, 3.0)),
            "tol": 1e-4 if m > 4000 else rng.choice([1e-4, 1e-6]), "fp64": fp64}


def _options(case):
    return PdlpOptions(verbose=False, primal_tol=case["tol"], dual_tol=case["tol"], optimality_tol=case["tol"],
                       enable_polishing=case["tol"] <= 1e-6,
                       precision=Precision.FP64 if case["fp64"] else Precision.Mixed)


def _known(m, n, seed):
    """A random sparse LP (rows alternating '=' and '<=', 0 <= x <= 10) and its
    optimal vertex: as many columns strictly inside their bounds as rows hold
    with equality, strict complementarity everywhere.  Returns (lp, x, y) with
    rc = c + A^T y the reduced costs."""
    lp, _ = G.random_lp(m, n, 4, 12, seed)
    rng = np.random.default_rng(seed)
    a = lp.matrix
    rows = np.repeat(np.arange(m), np.diff(a.row_starts))
    eq = np.arange(m) % 2 == 0
    tight = eq | (rng.random(m) < 0.5)
    x = np.where(rng.random(n) < 0.5, 0.0, 10.0)
    rc = np.where(x > 0.0, -1.0, 1.0) * rng.uniform(0.1, 1.0, n)
    inner = rng.choice(n, size=int(tight.sum()), replace=False)
    x[inner] = rng.uniform(1.0, 9.0, inner.size)
    rc[inner] = 0.0
    y = np.where(eq, rng.standard_normal(m), np.where(tight, rng.uniform(0.1, 1.0, m), 0.0))
    ax = np.bincount(rows, weights=a.values * x[a.col_indices], minlength=m)
    lp.row_upper = np.where(tight, ax, ax + rng.uniform(0.1, 1.0, m))
    lp.row_lower = np.where(eq, ax, -np.inf)
    lp.obj = rc - np.bincount(a.col_indices, weights=a.values * y[rows], minlength=n)
    return lp, x, y


def _lp(case, seed):
    if case["lp"] == "transport":
        return G.transport_lp(case["m"], case["n"], seed)[0]
    if case["lp"] == "powerlaw":
        return G.powerlaw_lp(case["m"], case["n"], seed=seed)[0]
    return _known(case["m"], case["n"], seed)[0]


def _batch_seeds(case, seed):
    sizes = G.batch_sizes(case["count"], median=float(case["median"]), lo=50, hi=6000, seed=5)
    return [(m, n, seed * 1009 + k) for k, (m, n) in enumerate(sizes)]


def prepare(case, seed):
    seed = int(seed) + 1
    kind, opts = case["kind"], _options(case)
    if kind == "batch":
        return kind, [_known(m, n, s)[0] for m, n, s in _batch_seeds(case, seed)], opts
    if kind == "serve":
        base, x0 = G.random_lp(case["m"], case["n"], 4, 12, seed)
        marks = G.integer_marks(case["n"], seed=seed)
        nodes = [G.node_lp(base, x0, marks, seed * 1009 + k, cuts_max=CUTS) for k in range(case["count"])]
        server = Server(opts, batch_window_ms=20)
        root = server.submit(base)
        server.wait(root)
        return kind, server, root, nodes, case["m"]
    lp = G.random_lp(case["m"], case["n"], 4, 12, seed)[0] if kind == "dive" else _lp(case, seed)
    if kind == "e2e":
        return kind, lp, opts
    solver = PdlpSolver()
    solver.setOptions(opts)
    solver.load(lp)
    if kind == "dive":
        solver.solve()
        x, y = solver.getPrimalValues(), solver.getDualValues()
        j = int(np.argmax(np.abs(x - np.round(x))))
        return kind, solver, x, y, j, float(np.floor(x[j]))
    return kind, solver


def _answer(result, x, y):
    return {"status": int(result.status), "iterations": int(result.iterations), "objective": float(result.objective),
            "x": x, "y": y}


def run(state):
    kind = state[0]
    if kind == "batch":
        out = batch_solve(state[1], state[2])
        return _joined(out)
    if kind == "serve":
        _, server, root, nodes, rows = state
        tickets = [server.submit(lp, warm=root) for lp in nodes]
        out = [server.wait(t) for t in tickets]
        for t in tickets:
            server.release(t)
        # a node appends up to CUTS rows of its own: the duals of all nodes as rows of one length
        return _joined([(r, x, np.pad(y, (0, rows + CUTS - y.size))) for r, x, y in out])
    if kind == "e2e":
        solver = PdlpSolver()
        solver.setOptions(state[2])
        solver.load(state[1])
    else:
        solver = state[1]
    if kind == "dive":
        _, _, x, y, j, bound = state
        solver.setColBounds(j, 0.0, bound)
        solver.setWarmStart(x, y)
    result = solver.solve()
    return _answer(result, solver.getPrimalValues(), solver.getDualValues())


def _joined(out):
    return {"status": np.array([int(r.status) for r, _, _ in out]),
            "iterations": np.array([int(r.iterations) for r, _, _ in out]),
            "objective": np.array([r.objective for r, _, _ in out]),
            "x": np.concatenate([x for _, x, _ in out]), "y": np.concatenate([y for _, _, y in out])}


def _sizes(case):
    """(rows, columns, nonzeros) of the case's LP or of its LPs together."""
    if case["kind"] == "batch":
        m = sum(s[0] for s in _batch_seeds(case, 1))
        return m, int(2.5 * m), int(20 * m)
    if case["lp"] == "transport":
        return case["m"] + case["n"], case["m"] * case["n"], 2 * case["m"] * case["n"]
    k = case.get("count", 1)
    return k * case["m"], k * case["n"], k * (10 if case["lp"] == "powerlaw" else 8) * case["n"]


def work(case):
    """One iteration multiplies by A and by A^T and updates every row and column.
    The number of iterations belongs to the data; these are round figures of
    what the tolerances take.  Where both matrix sides in FP32 and the vectors
    fit the chip's memory the matrix comes from HBM once, else each iteration
    reads it again."""
    m, n, nnz = _sizes(case)
    if case["lp"] == "transport":
        iters = 400 if case["tol"] > 0.05 else 20000 if case["tol"] < 5e-4 else 4000
    elif case["lp"] == "powerlaw":
        iters = 400 if case["tol"] > 0.05 else 800 if case["tol"] > 5e-3 else 2000
    elif case["kind"] in ("dive", "serve"):
        iters = 2000
    else:
        iters = 20000 if case["tol"] <= 1e-6 else 8000 if case["tol"] <= 1e-5 else 2000
    value = 8 if case["fp64"] else 4
    step = nnz * 2 * (4 + value) + (m + n) * 44
    once = nnz * 12 + (m + n) * 40 + 8 * (m + n)
    return {"bytes": float(iters * step if step > 126e6 else once), "flops": float(iters * (4 * nnz + 12 * (m + n)))}


def exact(case, seed):
    """The optimal vertex the LP was built around, where it was; its objective
    alone where the tolerance asks for an approximate answer, which need not be
    near the vertex."""
    seed = int(seed) + 1
    if case["lp"] != "random" or case["kind"] not in ("solve", "e2e", "batch"):
        return None
    near = case["tol"] <= 1e-6
    if case["kind"] == "batch":
        known = [_known(*s) for s in _batch_seeds(case, seed)]
        return {"status": np.zeros(len(known), dtype=np.int64), "iterations": None,
                "objective": np.array([float(lp.obj @ x) for lp, x, _ in known]),
                "x": np.concatenate([x for _, x, _ in known]) if near else None,
                "y": np.concatenate([y for _, _, y in known]) if near else None}
    lp, x, y = _known(case["m"], case["n"], seed)
    return {"status": 0, "iterations": None, "objective": float(lp.obj @ x), "x": x if near else None,
            "y": y if near else None}
