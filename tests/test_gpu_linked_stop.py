"""Stop requests and time limits end a solve after the restart cycle at hand.

The engine queues a linked cycle ahead of the host's look at the one before, which
may not cost a second cycle where a cycle is long (a large check frequency).
"""
import threading

import pytest

from mipx_b200 import generators as G
from mipx_b200.pdlp import PdlpOptions, PdlpSolver, Precision, Status, StopFlag

pytestmark = pytest.mark.gpu

N = 150000  # iterations per cycle: about 0.45 s of the linked cycle, 0.15 s of one block
NEVER = dict(verbose=False, primal_tol=1e-30, dual_tol=1e-30, optimality_tol=1e-30, enable_polishing=False,
             precision=Precision.FP64, termination_eval_frequency=N)


def _loaded(m, n):
    """A solver whose device image is built (the first solve does that)."""
    s = PdlpSolver()
    s.setOptions(PdlpOptions(**{**NEVER, "termination_eval_frequency": 10, "max_iter": 10}))
    s.load(G.random_lp(m, n, 4, 12, 5)[0])
    s.solve()
    return s


@pytest.mark.parametrize("m,n", [(2000, 5000), (60, 150)])
def test_time_limit(m, n):
    s = _loaded(m, n)
    s.setOptions(PdlpOptions(max_solve_seconds=0.08, **NEVER))
    r = s.solve()
    assert (r.status, r.iterations) == (Status.TimeLimit, N)


@pytest.mark.parametrize("m,n", [(2000, 5000), (60, 150)])
def test_stop_flag(m, n):
    s, flag = _loaded(m, n), StopFlag()
    s.setOptions(PdlpOptions(stop_flag=flag, **NEVER))
    t = threading.Timer(0.08, flag.set)
    t.start()
    r = s.solve()
    t.join()
    assert (r.status, r.iterations) == (Status.IterLimit, N)
