"""The three forms of a pack's restart cycle -- step launches, linked, persistent -- give
the same bits, with LPs finishing at different times and dropped from the launches.

Pinned launch shapes keep the step launches; 17 and 18 (sliced ELL, 4 and 8 entries
per round) are the ones that 8 entries per column and 20 per row get anyway.
"""
import numpy as np
import pytest

from mipx_b200 import generators as G
from mipx_b200.pdlp import PdlpOptions, Precision, Server, batch_solve

pytestmark = pytest.mark.gpu

OPTS = dict(verbose=False, primal_tol=1e-5, dual_tol=1e-5, optimality_tol=1e-5, enable_polishing=False, max_iter=30000)
LAUNCHES = dict(shape_primal=17, shape_dual=18)
FIELDS = ("status", "iterations", "restarts", "objective", "primal_objective", "dual_objective", "rel_primal_resid",
          "rel_dual_resid", "primal_weight", "step_size", "fp64_iterations")


def _lps():
    sizes = (33, 257, 300, 700, 1013, 2100, 60, 450)
    return [G.random_lp(m, int(2.5 * m), 4, 12, 80 + m)[0] for m in sizes]


def _same(a, b):
    for (r, x, y), (q, u, v) in zip(a, b):
        for f in FIELDS:
            assert getattr(r, f) == getattr(q, f), f
        np.testing.assert_array_equal(x, u)
        np.testing.assert_array_equal(y, v)


@pytest.mark.parametrize("precision", [Precision.Mixed, Precision.FP64])
@pytest.mark.parametrize("compact", [True, False])
def test_three_forms(precision, compact):
    lps = _lps()
    o = dict(OPTS, precision=precision, batch_compact=compact)
    launches = batch_solve(lps, PdlpOptions(**o, **LAUNCHES))
    linked = batch_solve(lps, PdlpOptions(**o))
    persistent = batch_solve(lps, PdlpOptions(**o, batch_persistent=True))
    _same(launches, linked)
    _same(launches, persistent)
    # each form ran: per cycle the steps take 2 x 200 launches, two, one
    cycles = max(r.iterations for r, _, _ in launches) / 200
    n = [max(r.kernel_launches for r, _, _ in a) for a in (launches, linked, persistent)]
    assert n[0] - n[1] >= 390 * cycles
    assert 0.5 * cycles <= n[1] - n[2] <= 1.5 * cycles


def test_server_packs():
    lps = _lps()
    out = []
    for pins in (LAUNCHES, {}):
        with Server(PdlpOptions(**OPTS, **pins), batch_window_ms=50) as srv:
            tickets = [srv.submit(lp) for lp in lps]
            out.append([srv.wait(t) for t in tickets])
    _same(*out)
