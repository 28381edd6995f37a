"""Options changed between two solves of one loaded LP.

The engine keeps its captured graphs from solve to solve; what a graph holds by value
-- iteration limits, the power iteration's limit and tolerance, Anderson's
regularisation -- has to be that of the solve at hand.  Compared with a new solver.
"""
import numpy as np
import pytest

from mipx_b200 import generators as G
from mipx_b200.pdlp import PdlpOptions, PdlpSolver, Status

pytestmark = pytest.mark.gpu

BASE = dict(verbose=False, primal_tol=1e-6, dual_tol=1e-6, optimality_tol=1e-6, enable_polishing=True,
            polish_primal_tol=1e-9, polish_dual_tol=1e-9, max_iter=100000, polish_max_iter=1000)
FIELDS = ("status", "iterations", "restarts", "objective", "primal_objective", "dual_objective", "rel_primal_resid",
          "rel_dual_resid", "primal_weight", "step_size")


# one block, linked cycle, step launches
@pytest.mark.parametrize("m,n,pins", [(60, 150, {}), (400, 1000, {}), (400, 1000, dict(shape_primal=17, shape_dual=17))])
@pytest.mark.parametrize("first,second", [(dict(max_iter=600), dict()), (dict(), dict(max_iter=600)),
                                          (dict(polish_max_iter=200), dict()),
                                          (dict(sv_max_iter=2), dict()), (dict(sv_tol=0.3), dict()),
                                          (dict(anderson_acceleration=True, anderson_regularization=0.5),
                                           dict(anderson_acceleration=True))])
def test_second_solve_has_the_second_options(m, n, pins, first, second):
    lp, _ = G.random_lp(m, n, 4, 12, 21)
    s, t = PdlpSolver(), PdlpSolver()
    s.setOptions(PdlpOptions(**{**BASE, **pins, **first}))
    s.load(lp)
    s.solve()
    s.setOptions(PdlpOptions(**{**BASE, **pins, **second}))
    a = s.solve()
    t.setOptions(PdlpOptions(**{**BASE, **pins, **second}))
    t.load(lp)
    b = t.solve()
    for f in FIELDS:
        assert getattr(a, f) == getattr(b, f), f
    if b.status != Status.Optimal:  # a solve that ends at its limit leaves x and y as they were
        return
    np.testing.assert_array_equal(s.getPrimalValues(), t.getPrimalValues())
    np.testing.assert_array_equal(s.getDualValues(), t.getDualValues())
