"""The bounded waits of the linked restart cycle (csrc/linked.cuh) run out.

With a limit of one load per wait (option link_polls) the first value that is not
there yet ends the cycle: every warp leaves, the call returns PDLPX_E_TIMEOUT, and
the same solver, and the next batch, solve as if nothing had been.
"""
import numpy as np
import pytest

from mipx_b200 import _capi
from mipx_b200 import generators as G
from mipx_b200.pdlp import PdlpOptions, PdlpSolver, Precision, Status, batch_solve

pytestmark = pytest.mark.gpu

OPTS = dict(verbose=False, primal_tol=1e-4, dual_tol=1e-4, optimality_tol=1e-4, enable_polishing=False)
TIMEOUT = 6


def _lp(kind):
    if kind == "csr":
        return G.transport_lp(97, 131, 3)[0]
    if kind == "long":
        return G.powerlaw_lp(1500, 6000, kmax=300, seed=4)[0]
    return G.random_lp(2000, 5000, 4, 12, 5)[0]


@pytest.mark.parametrize("kind", ["sell", "csr", "long"])
def test_single_lp(kind):
    s, t = PdlpSolver(), PdlpSolver()
    for k in (s, t):
        k.setOptions(PdlpOptions(**OPTS))
        k.load(_lp(kind))
    for _ in range(2):
        s.setOptions(PdlpOptions(link_polls=1, **OPTS))
        with pytest.raises(_capi.PdlpxError, match="timed out") as e:
            s.solve()
        assert e.value.code == TIMEOUT
        assert s.getStatus() == Status.Error
        s.setOptions(PdlpOptions(**OPTS))
        a, b = s.solve(), t.solve()
        assert (a.status, a.iterations, a.objective) == (b.status, b.iterations, b.objective)
        np.testing.assert_array_equal(s.getPrimalValues(), t.getPrimalValues())
        np.testing.assert_array_equal(s.getDualValues(), t.getDualValues())


@pytest.mark.parametrize("precision", [Precision.Mixed, Precision.FP64])
def test_pack(precision):
    lps = [G.random_lp(m, int(2.5 * m), 4, 12, 70 + m)[0] for m in (300, 900, 2500)]
    want = batch_solve(lps, PdlpOptions(precision=precision, **OPTS))
    with pytest.raises(_capi.PdlpxError, match="timed out") as e:
        batch_solve(lps, PdlpOptions(precision=precision, link_polls=1, **OPTS))
    assert e.value.code == TIMEOUT
    for (r, x, y), (q, u, v) in zip(batch_solve(lps, PdlpOptions(precision=precision, **OPTS)), want):
        assert (r.status, r.iterations, r.objective) == (q.status, q.iterations, q.objective)
        np.testing.assert_array_equal(x, u)
        np.testing.assert_array_equal(y, v)


def test_one_block_waits_for_nothing():
    s = PdlpSolver()
    s.setOptions(PdlpOptions(link_polls=1, **OPTS))
    s.load(G.random_lp(60, 150, 4, 12, 2)[0])
    assert s.solve().status == Status.Optimal
