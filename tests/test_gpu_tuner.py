"""The smoother's tuner on a forest solved with one state per problem: after a
solve, when every problem is finished and the sweeps would leave all of them
alone, it still times sweeps that do their work, and the states of the last
solve can still be asked for."""
import numpy as np
import pytest

from sayakaamr_gb300 import workloads as W

pytestmark = pytest.mark.gpu

PARAMS = dict(tol_rel=1e-8, tol_abs=0.0, use_mg_precond=1, bottom=1, max_iter=500)


@pytest.mark.parametrize("first, second", [(1, 0), (0, 1)])
def test_times_after_a_solve_are_those_of_a_fresh_solver(first, second):
    p = W.config4(n_problems=128)
    S = W.make_solver(p, precision=first, **PARAMS)
    S.cg_solve()
    before = S.problem_states()
    S.set_params(precision=second)
    S.prepare()
    after = S.problem_states()
    T = W.make_solver(p, precision=second, **PARAMS)
    T.prepare()
    # 17 M cells: a sweep takes several times as long as a launch that does nothing
    late, fresh = np.array(S.tuned_smoother(second)[1]), np.array(T.tuned_smoother(second)[1])
    assert np.median(late / fresh) > 0.7, (late, fresh)
    assert np.array_equal(before[0], after[0]) and np.array_equal(before[1], after[1])
