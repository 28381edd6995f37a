"""Family packs whose members have rows with two finite sides, in the base and among
the appended rows: the same bits alone and among others, for every form of the steps
(appended rows by lane or by column, one or several columns and rows per warp).
"""
import numpy as np
import pytest

from mipx_b200 import generators as G
from mipx_b200.pdlp import PdlpOptions, Server

pytestmark = pytest.mark.gpu

OPTS = dict(verbose=False, primal_tol=1e-4, dual_tol=1e-4, optimality_tol=1e-4, enable_polishing=False, max_iter=4000)


def _ranged(lp, seed):
    rng = np.random.default_rng(seed)
    lo = np.where(np.isfinite(lp.row_lower), lp.row_lower, lp.row_upper - rng.uniform(0.5, 5.0, lp.num_rows))
    hi = np.where(np.isfinite(lp.row_upper), lp.row_upper, lp.row_lower + rng.uniform(0.5, 5.0, lp.num_rows))
    some = rng.random(lp.num_rows) < 0.6
    lp.row_lower = np.where(some, np.minimum(lo, hi - 0.3), lp.row_lower)
    lp.row_upper = np.where(some, hi, lp.row_upper)
    return lp


@pytest.mark.parametrize("m,n,count,cuts", [(130, 333, 32, 0), (130, 333, 9, 50), (300, 750, 32, 50), (6000, 15000, 6, 20)])
def test_alone_and_together(m, n, count, cuts):
    base, x0 = G.random_lp(m, n, 3, 9, 5)
    base = _ranged(base, 1)
    marks = G.integer_marks(n)
    nodes = [_ranged(G.node_lp(base, x0, marks, 900 + k, cuts_max=cuts, cut_nnz=(20, 200)), k) for k in range(count)]
    with Server(PdlpOptions(**OPTS), batch_window_ms=50) as srv:
        root = srv.submit(base)
        srv.wait(root)
        tickets = [srv.submit(lp, warm=root) for lp in nodes]
        together = [srv.wait(t) for t in tickets]
        alone = [srv.wait(srv.submit(lp, warm=root)) for lp in nodes[:4]]
    for (r, x, y), (q, u, v) in zip(alone, together):
        assert (r.status, r.iterations, r.objective) == (q.status, q.iterations, q.objective)
        assert (r.rel_primal_resid, r.rel_dual_resid) == (q.rel_primal_resid, q.rel_dual_resid)
        np.testing.assert_array_equal(x, u)
        np.testing.assert_array_equal(y, v)
