"""An asynchronous solve without a captured graph takes its parameters as they
are when it is enqueued: with the double-float operator or the learned
correction switched on after the preparation it gives the bits of a solver that
was prepared with them, also where the arrays that only they read had been
built from other coefficients."""
import numpy as np
import pytest

from oracle import nn_oracle as nn
from sayakaamr_gb300 import workloads as W

pytestmark = pytest.mark.gpu

PARAMS = dict(tol_rel=1e-8, tol_abs=0.0, use_mg_precond=1, bottom=1, precision=1, max_iter=200, graph=0)


def _scale_b(S, p, a):
    for d in range(p.ndim):
        S.set_coef_b(d, a * np.asarray(p.bface[d]))


# (the correction's own buffers are made by a preparation that has it on)
@pytest.mark.parametrize("late, other_coefficients",
                         [(dict(vcycle_out=1), False), (dict(vcycle_out=1), True), (dict(learned=1), True)],
                         ids=["double-float-unbuilt", "double-float-stale", "learned-stale"])
def test_parameters_set_after_the_preparation(late, other_coefficients):
    p = W.config2(nb=8, max_level=4)
    weights = nn.init(8)
    S, T = W.make_solver(p, **PARAMS), W.make_solver(p, **PARAMS)
    for s in (S, T):
        s.set_learned_weights(weights)
    if other_coefficients:
        _scale_b(S, p, 3.0)
        S.set_params(**late)
        S.cg_solve()
        S.set_params(**{k: 0 for k in late})
        _scale_b(S, p, 1.0)
    S.prepare()
    S.set_zero_sol()
    S.set_params(**late)
    S.cg_solve_async()
    a = S.solve_info()
    T.set_params(**late)
    b = T.cg_solve()
    assert b["rnorm"] < 1e-8 * b["rnorm0"], b
    assert (a["status"], a["iterations"], a["rnorm"]) == (b["status"], b["iterations"], b["rnorm"])
    assert np.array_equal(S.get_sol_compact(), T.get_sol_compact())
