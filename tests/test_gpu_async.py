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


def _disk(seed):
    """fluid inside a disk only: more than a quarter of the blocks is solid"""
    t = W.refine_tree(2, 8, (2, 2, 1), (0, 0, 0), (1, 1, 0), 3, 5,
                      lambda lo, hi, l: np.abs(np.hypot(*(0.5 * (lo + hi) - [0.45, 0.8]).T) - 0.2) < 1.2 * (hi - lo)[:, 0])
    tb = t.tables()
    d = lambda p: 0.2 - np.hypot(p[..., 0] - 0.45, p[..., 1] - 0.82)  # noqa: E731
    vol = (d(W.cell_centres(tb)) > 0).astype(np.float64)
    area = [(d(W.face_centres(tb, q)) > 0).astype(np.float64) for q in range(2)]
    f = W.gaussian_rhs(np.random.default_rng(seed), W.cell_centres(tb), 2)
    p = W._finish("disk", t, tb, vol, area, [np.ones_like(a) for a in area], f, False, {}, dirichlet_faces=(3,))
    assert 4 * (p.vol.reshape(p.num_blocks, -1).max(axis=1) == 0).sum() > p.num_blocks
    return p


@pytest.mark.parametrize("early, late", [(dict(learned=0), dict(learned=1)), (dict(per_problem=0), dict(per_problem=1))],
                         ids=["learned", "per-problem"])
def test_mostly_solid_domain(early, late):
    learned = "learned" in late
    p = _disk(3) if learned else W.forest([_disk(3), _disk(4)], "disks")
    weights = nn.init(8)
    S, T = W.make_solver(p, **PARAMS), W.make_solver(p, **PARAMS)
    for s in (S, T):
        if learned:
            s.set_learned_weights(weights)
        # (the correction's own buffers are made by a preparation that has it on)
        s.set_params(**late)
        s.cg_solve()
        s.set_zero_sol()
    S.set_params(**early)
    S.prepare()
    S.set_params(**late)
    S.cg_solve_async()
    a = S.solve_info()
    b = T.cg_solve()
    assert b["rnorm"] < 1e-8 * b["rnorm0"], b
    assert (a["status"], a["iterations"], a["rnorm"]) == (b["status"], b["iterations"], b["rnorm"])
    assert np.array_equal(S.get_sol_compact(), T.get_sol_compact())
