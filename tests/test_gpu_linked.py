"""The linked restart cycle (csrc/linked.cuh) against the step launches.

Both sum every row in the same order and update it by the same expressions, so
iterations, objective, x and y are the same bits.  The launches run where a
launch shape is pinned; a pinned sliced-ELL variant (17: 4 entries per round)
or the row-length table's own CSR shape (10: 32 lanes) changes no sum.
"""
import threading

import numpy as np
import pytest

from mipx_b200 import generators as G
from mipx_b200.pdlp import LpProblem, PdlpOptions, PdlpSolver, Precision, SparseMatrix, batch_solve

pytestmark = pytest.mark.gpu

LOOSE = dict(verbose=False, primal_tol=1e-4, dual_tol=1e-4, optimality_tol=1e-4, enable_polishing=False)

# of the last check, so they tell the iterates apart where a capped solve returns no x
FIELDS = ("status", "iterations", "restarts", "objective", "primal_objective", "dual_objective", "rel_primal_resid",
          "rel_dual_resid", "primal_weight", "step_size", "fp64_iterations")


def _solve(lp, **kw):
    s = PdlpSolver()
    s.setOptions(PdlpOptions(**{**LOOSE, **kw}))
    s.load(lp)
    r = s.solve()
    return r, s


def _same(lp, pins, **kw):
    a, sa = _solve(lp, **kw)
    b, sb = _solve(lp, **pins, **kw)
    assert a.kernel_launches < b.kernel_launches, "the linked cycle did not run"
    for f in FIELDS:
        assert getattr(a, f) == getattr(b, f), f
    np.testing.assert_array_equal(sa.getPrimalValues(), sb.getPrimalValues())
    np.testing.assert_array_equal(sa.getDualValues(), sb.getDualValues())


SELL = dict(shape_primal=17, shape_dual=17)


def _holes(m, n, seed):
    """Rows and columns without entries among rows of 0-40 entries."""
    rng = np.random.default_rng(seed)
    lens = np.where(rng.random(m) < 0.3, 0, rng.integers(1, min(n, 40) + 1, m))
    ci = [np.sort(rng.choice(max(1, n - 3), size=min(k, max(1, n - 3)), replace=False)) for k in lens]
    rp = np.concatenate([[0], np.cumsum([c.size for c in ci])]).astype(np.int32)
    ci = np.concatenate(ci + [np.zeros(0, int)]).astype(np.int32)
    v = rng.standard_normal(ci.size)
    x0 = rng.uniform(0, 10, n)
    ax = np.zeros(m)
    np.add.at(ax, np.repeat(np.arange(m), np.diff(rp)), v * x0[ci])
    return LpProblem(num_cols=n, num_rows=m, obj=rng.standard_normal(n), col_lower=np.zeros(n),
                     col_upper=np.full(n, 10.0), row_lower=np.where(np.arange(m) % 3 == 0, ax, -np.inf),
                     row_upper=ax + np.where(np.arange(m) % 3 == 0, 0.0, 1.0),
                     matrix=SparseMatrix(m, n, values=v, col_indices=ci, row_starts=rp))


# sizes around a warp's rows with 2, 4 and 8 lanes per row and around a slice,
# columns longer than rows, one-entry LPs, and more units than the grid has warps
@pytest.mark.parametrize("m,n,lo,hi", [(1, 1, 1, 1), (3, 7, 1, 2), (8, 9, 1, 8), (31, 33, 2, 9), (33, 64, 4, 12),
                                       (257, 640, 4, 12), (900, 300, 18, 40), (1013, 2531, 4, 12), (5000, 12500, 1, 3),
                                       (14000, 35000, 4, 12)])
@pytest.mark.parametrize("precision", [Precision.FP64, Precision.Mixed])
def test_sliced_ell(m, n, lo, hi, precision):
    lp, _ = G.random_lp(m, n, lo, hi, 40 + m)
    _same(lp, SELL, precision=precision, fp64_switch=precision == Precision.FP64, max_iter=1500)


# one block: 12 slices and 13, up to 16 entries on one side and 40 on the other
# (and one more), either side the short one, rows with two finite sides
@pytest.mark.parametrize("m,n,lo,hi", [(32, 352, 1, 3), (33, 352, 1, 3), (352, 32, 20, 32), (240, 120, 8, 30),
                                       (90, 250, 4, 16), (90, 250, 4, 17), (60, 150, 12, 16), (41, 41, 40, 41)])
@pytest.mark.parametrize("precision", [Precision.FP64, Precision.Mixed])
@pytest.mark.parametrize("ranged", [False, True])
def test_one_block(m, n, lo, hi, precision, ranged):
    lp, _ = G.random_lp(m, n, lo, hi, 7 + m)
    if ranged:
        hi_side = np.where(np.isfinite(lp.row_upper), lp.row_upper, lp.row_lower + 1.0)
        lo_side = np.where(np.isfinite(lp.row_lower), lp.row_lower, lp.row_upper - 1.0)
        lp.row_lower, lp.row_upper = np.minimum(lo_side, hi_side - 0.5), hi_side
    _same(lp, SELL, precision=precision, max_iter=1500)
    _same(lp, SELL, precision=precision, fp64_switch=False, max_iter=450)


@pytest.mark.parametrize("m,n", [(5, 40), (64, 50), (700, 900)])
def test_empty_rows_and_columns(m, n):
    _same(_holes(m, n, m), SELL, max_iter=1000)


@pytest.mark.parametrize("s,d", [(70, 80), (97, 131), (130, 180), (200, 210)])
@pytest.mark.parametrize("fp32", [False, True])
def test_csr_rows(s, d, fp32):
    lp, _ = G.transport_lp(s, d, 3)
    pins = dict(shape_primal=17, shape_dual=10 if lp.matrix.numNonzeros() / (s + d) <= 128 else 12)
    _same(lp, pins, fp64_switch=not fp32, max_iter=1000)


@pytest.mark.parametrize("m,kmax", [(1500, 100), (1500, 300), (3000, 700), (3000, 1000)])
def test_long_columns(m, kmax):
    lp, _ = G.powerlaw_lp(m, 4 * m, kmax=kmax, seed=m + kmax)
    _same(lp, SELL, max_iter=1000)
    _same(lp, SELL, max_iter=600, fp64_switch=False)


# cycles cut short by the iteration limit, one iteration per cycle, restarts that
# write y between cycles, the FP32 -> FP64 hand-over and the polish phase
@pytest.mark.parametrize("kw", [dict(max_iter=777), dict(termination_eval_frequency=1, max_iter=60),
                                dict(termination_eval_frequency=7, max_iter=400), dict(adaptive_step=True),
                                dict(anderson_acceleration=True), dict(precision=Precision.FP64),
                                dict(primal_tol=1e-5, dual_tol=1e-5, optimality_tol=1e-5, enable_polishing=True)])
def test_cycles(kw):
    lp, _ = G.random_lp(400, 1000, 4, 12, 8)
    _same(lp, SELL, **kw)


def test_repeated_solves_and_warm_start():
    lp, _ = G.random_lp(300, 800, 4, 12, 9)
    r, s = _solve(lp)
    x, y = s.getPrimalValues(), s.getDualValues()
    q = s.solve()
    assert (q.iterations, q.objective) == (r.iterations, r.objective)
    np.testing.assert_array_equal(s.getPrimalValues(), x)
    s.setWarmStart(x, y)
    w = s.solve()
    _, t = _solve(lp, **SELL)
    t.setWarmStart(x, y)
    v = t.solve()
    assert (w.iterations, w.objective) == (v.iterations, v.objective)
    np.testing.assert_array_equal(s.getPrimalValues(), t.getPrimalValues())


def test_many_threads():
    """More waiting grids than the SMs hold: every solve ends with the bits it has alone."""
    lp, _ = G.random_lp(2000, 5000, 4, 12, 5)
    alone, s = _solve(lp)
    out = [None] * 12

    def go(k):
        r, t = _solve(lp)
        out[k] = (r.iterations, r.objective, t.getDualValues())

    ts = [threading.Thread(target=go, args=(k,)) for k in range(len(out))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    y = s.getDualValues()
    for r in out:
        assert r is not None and r[:2] == (alone.iterations, alone.objective)
        np.testing.assert_array_equal(r[2], y)


# packs: the persistent cycle runs the step kernels' own tile functions
@pytest.mark.parametrize("kw", [dict(), dict(precision=Precision.FP64), dict(max_iter=777), dict(batch_compact=False),
                                dict(termination_eval_frequency=7, max_iter=300),
                                dict(primal_tol=1e-6, dual_tol=1e-6, optimality_tol=1e-6, enable_polishing=True)])
def test_packs(kw):
    lps = [G.random_lp(m, n, lo, hi, 60 + m)[0] for m, n, lo, hi in
           ((1, 1, 1, 1), (3, 7, 1, 2), (31, 33, 2, 9), (257, 640, 4, 12), (256, 256, 4, 30), (700, 1750, 4, 12),
            (2100, 5000, 4, 12))] + [_holes(64, 50, 2)]
    rng = np.random.default_rng(0)
    warm = [None] * (len(lps) - 1) + [(rng.uniform(0, 1, 50), rng.standard_normal(64))]
    a = batch_solve(lps, PdlpOptions(**{**LOOSE, **kw}), warm=warm)
    b = batch_solve(lps, PdlpOptions(batch_persistent=True, **{**LOOSE, **kw}), warm=warm)
    for (r, x, y), (q, u, v) in zip(a, b):
        for f in FIELDS:
            assert getattr(r, f) == getattr(q, f), f
        np.testing.assert_array_equal(x, u)
        np.testing.assert_array_equal(y, v)


def test_packs_from_many_threads():
    lps = [G.random_lp(m, int(2.5 * m), 4, 12, 70 + m)[0] for m in (300, 900, 1500, 2500, 4000)]
    alone = batch_solve(lps, PdlpOptions(**LOOSE))
    out = [None] * 6
    ts = [threading.Thread(target=lambda k=k: out.__setitem__(k, batch_solve(lps, PdlpOptions(**LOOSE))))
          for k in range(len(out))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for res in out:
        for (r, x, y), (q, u, v) in zip(alone, res):
            assert (r.iterations, r.objective) == (q.iterations, q.objective)
            np.testing.assert_array_equal(x, u)
            np.testing.assert_array_equal(y, v)


# long and short columns of the primal step in one launch, against the two launches
# that a pinned sliced-ELL variant other than the table's takes (19: 16 entries per round)
@pytest.mark.parametrize("m,kmax,kmean", [(9000, 90, 10.0), (9000, 2000, 10.0), (6000, 6000, 30.0)])
@pytest.mark.parametrize("precision", [Precision.Mixed, Precision.FP64])
def test_long_and_short_columns_in_one_launch(m, kmax, kmean, precision):
    lp, _ = G.powerlaw_lp(m, 4 * m + 5, kmax=kmax, kmean=kmean, seed=m + kmax)
    pins = dict(shape_dual=18, precision=precision, max_iter=400, termination_eval_frequency=100)
    a, sa = _solve(lp, shape_primal=17, **pins)
    b, sb = _solve(lp, shape_primal=19, **pins)
    assert a.kernel_launches < b.kernel_launches, "the launches did not run as one"
    for f in FIELDS:
        assert getattr(a, f) == getattr(b, f), f
