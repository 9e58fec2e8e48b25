"""The bounded waits of the one-launch smoothing: a wait for a block that is
not there runs out, the call reports it and the device goes on; a solve that
finds the error word set ends after the iteration it is in, whatever its limit
and tolerance, and reports it."""
import ctypes as C

import pytest

import sayakaamr_gb300 as sg
from sayakaamr_gb300 import workloads as W
from test_gpu_active import _tube
from test_gpu_async import _disk

pytestmark = pytest.mark.gpu

# a tolerance out of reach: a solve that does not look at the word runs to max_iter
PARAMS = dict(tol_rel=1e-30, tol_abs=0.0, use_mg_precond=1, bottom=1, precision=1, max_iter=300)


def _solves(p):
    S = W.make_solver(p, **dict(PARAMS, tol_rel=1e-8))
    info = S.cg_solve()
    assert info["rnorm"] < 1e-8 * info["rnorm0"], info


@pytest.mark.parametrize("p", [lambda: W.config2(nb=16, max_level=4), lambda: W.config2(nb=8, max_level=4),
                               lambda: _tube(5.0)], ids=["2d-16", "2d-8", "3d-8"])
def test_a_wait_that_runs_out(p):
    p = p()
    assert len(set(p.tables["level"][p.leaf])) > 1  # both parity groups
    S = W.make_solver(p, **PARAMS)
    with pytest.raises(RuntimeError, match="bounded wait"):
        S.fail_wait(int(p.tables["level"].max()), 2000)
    _solves(p)


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("p", [lambda: W.config2(nb=8, max_level=4), lambda: W.forest([_disk(3), _disk(4)], "disks"),
                               lambda: W.config3(nb=8, max_level=3, band=1.0)], ids=["2d", "forest", "3d"])
def test_a_solve_ends_after_the_iteration(p, graph):
    p = p()
    S = W.make_solver(p, graph=graph, **PARAMS)
    S.prepare()
    S.set_wait_error()
    with pytest.raises(RuntimeError, match="bounded wait"):
        S.cg_solve()
    info = sg.SolveInfo()
    S.lib.sayaka_mac_solve_info(S.h, C.byref(info))
    assert info.iterations <= 1
    _solves(p)
