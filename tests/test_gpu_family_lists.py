"""Appended rows of a family pack's members by lane and by column.

A pack whose members append many rows walks them by lane, a pack of one or two
members by column; one or several columns / rows per warp by the base's size.
A member's sums have the same order either way, so its result is the same bits
alone and among others.
"""
import numpy as np
import pytest

from mipx_b200 import generators as G
from mipx_b200.pdlp import PdlpOptions, Server

pytestmark = pytest.mark.gpu

OPTS = dict(verbose=False, primal_tol=1e-4, dual_tol=1e-4, optimality_tol=1e-4, enable_polishing=False)


# a base of one warp's columns, ragged ones, and one beyond 32 columns per SM and warp slot
@pytest.mark.parametrize("m,n,count,cuts", [(12, 31, 3, 6), (130, 333, 32, 0), (130, 333, 9, 50), (300, 750, 32, 50),
                                            (2100, 5300, 5, 50)])
def test_alone_and_together(m, n, count, cuts):
    base, x0 = G.random_lp(m, n, 3, 9, 5)
    marks = G.integer_marks(n)
    nodes = [G.node_lp(base, x0, marks, 900 + k, cuts_max=cuts, cut_nnz=(min(n, 20), min(n, 200))) for k in range(count)]
    with Server(PdlpOptions(**OPTS), batch_window_ms=50) as srv:
        root = srv.submit(base)
        srv.wait(root)
        tickets = [srv.submit(lp, warm=root) for lp in nodes]
        together = [srv.wait(t) for t in tickets]
        alone = []
        for lp in nodes[:4]:
            t = srv.submit(lp, warm=root)
            alone.append(srv.wait(t))
    for (r, x, y), (q, u, v) in zip(alone, together):
        assert (r.status, r.iterations, r.objective) == (q.status, q.iterations, q.objective)
        np.testing.assert_array_equal(x, u)
        np.testing.assert_array_equal(y, v)
