"""The FP32 -> FP64 hand-over with the linked restart cycle (csrc/linked.cuh).

The engine queues the next cycle before it has read that the one at hand handed the
iterates to FP64, so one FP32 cycle runs that must change nothing.  Compared with
the step launches, which are queued one at a time and give the same bits.
"""
import numpy as np
import pytest

from mipx_b200.pdlp import LpProblem, PdlpOptions, PdlpSolver, Precision, SparseMatrix

pytestmark = pytest.mark.gpu

FIELDS = ("status", "iterations", "fp64_iterations", "restarts", "objective", "primal_objective", "dual_objective",
          "rel_primal_resid", "rel_dual_resid", "rel_gap", "primal_weight", "step_size")
TOL = dict(verbose=False, primal_tol=1e-3, dual_tol=1e-3, optimality_tol=1e-3, enable_polishing=False)
LAUNCHES = dict(shape_primal=17, shape_dual=17)  # a pinned shape keeps the step launches


@pytest.fixture(scope="module")
def lp():
    """Large enough for FP32 (16 MiB of matrix and vectors), small enough to be linked
    (560,000 entries), and soon at FP32's rounding: the entries of a row come in pairs
    v, -v and the columns lie in [1e5, 1e5 + 10], so activities are differences of
    numbers 10,000 times as large."""
    m, n, pairs, shift = 28000, 70000, 10, 1e5
    rng = np.random.default_rng(3)
    ci = np.stack([np.sort(rng.choice(n, 2 * pairs, replace=False)) for _ in range(m)])
    v = rng.standard_normal((m, pairs))
    v = np.stack([v, -v], axis=2).reshape(m, 2 * pairs)
    ax = (v * rng.uniform(0, 10, n)[ci]).sum(1)
    eq = np.arange(m) % 2 == 0
    return LpProblem(num_cols=n, num_rows=m, obj=rng.standard_normal(n), col_lower=np.full(n, shift),
                     col_upper=np.full(n, shift + 10.0), row_lower=np.where(eq, ax, -np.inf),
                     row_upper=np.where(eq, ax, ax + 1.0),
                     matrix=SparseMatrix(m, n, values=v.ravel(), col_indices=ci.ravel().astype(np.int32),
                                         row_starts=(2 * pairs * np.arange(m + 1)).astype(np.int32)))


@pytest.fixture(scope="module")
def warm(lp):
    s = PdlpSolver()
    s.setOptions(PdlpOptions(precision=Precision.FP64, **TOL))
    s.load(lp)
    s.solve()
    return s.getPrimalValues(), s.getDualValues()


# a restart at every check, the hand-over's among them, and the ordinary rules
@pytest.mark.parametrize("fraction", [0.0, 0.05])
@pytest.mark.parametrize("anderson", [False, True])
@pytest.mark.parametrize("adaptive", [False, True])
def test_same_bits_as_the_launches(lp, warm, fraction, anderson, adaptive):
    out = []
    for pins in ({}, LAUNCHES):
        s = PdlpSolver()
        s.setOptions(PdlpOptions(max_iter=4000, termination_eval_frequency=40, restart_artificial_fraction=fraction,
                                 anderson_acceleration=anderson, adaptive_step=adaptive, **TOL, **pins))
        s.load(lp)
        s.setWarmStart(*warm)
        r = s.solve()
        out.append((r, s.getPrimalValues(), s.getDualValues()))
    (a, x, y), (b, u, v) = out
    assert a.kernel_launches < b.kernel_launches, "the linked cycle did not run"
    if not adaptive:
        assert 0 < b.fp64_iterations < b.iterations, "no hand-over on the way"
    for f in FIELDS:
        assert getattr(a, f) == getattr(b, f), f
    np.testing.assert_array_equal(x, u)
    np.testing.assert_array_equal(y, v)
