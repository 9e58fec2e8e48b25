"""That the one-launch smoothing is what runs where a tower fits: fewer launches an
iteration than with separate ones, other towers as the body moves, and none of it
where no tower fits; and the sweeps' launch variants, which such towers do not
take, compared where they run (prolong_form 0)."""
import numpy as np
import pytest

from sayakaamr_gb300 import workloads as W
from test_gpu_active import _tube
from test_gpu_parity import setup_solver

pytestmark = pytest.mark.gpu

PARAMS = dict(tol_rel=1e-8, tol_abs=0.0, use_mg_precond=1, bottom=1, precision=1, max_iter=500)


def _launches(S, form):
    S.set_params(prolong_form=form)
    S.prepare()
    return S.launch_counts()[1]


@pytest.mark.parametrize("problem", [lambda: W.config2(nb=16, max_level=5), lambda: W.config2(nb=8, max_level=5),
                                     lambda: _tube(5.0)], ids=["2d-16", "2d-8", "3d-8"])
def test_every_tower_in_one_launch(problem):
    p = problem()
    S = W.make_solver(p, **PARAMS)
    one, separate = _launches(S, 1), _launches(S, 0)
    towers = int(p.tables["level"].max()) - S.bottom_level()
    # two sweeps of a tower over two parity groups: the fused prolongation and
    # seven colour launches at most, at least three; twice an iteration
    assert 2 * 2 * towers <= separate - one <= 2 * 7 * towers
    assert S.cg_solve()["status"] == 0


def test_the_finest_tower_does_not_fit():
    p = W.config2(nb=8, max_level=8)
    S = W.make_solver(p, **PARAMS)
    sizes = [S.tower_size(L) for L in range(2, 9)]
    assert sizes[0] < 152 * 8 and sizes[-1] > 152 * 16
    assert _launches(S, 1) < _launches(S, 0)


def test_no_tower_of_another_side_fits():
    S = W.make_solver(W.config2(nb=4, max_level=4), **PARAMS)
    assert _launches(S, 1) == _launches(S, 0)


def test_other_towers_fit_after_the_body_moves():
    """the finest towers fit while the pipe is mostly solid and not once all of it
    is fluid; the bits are those of separate launches before and after"""
    p = next(iter(W.config5_sequence(steps=1, regrid_every=100, max_level=6)))[2]
    out = []
    for form in (1, 0):
        S = W.make_solver(p, **dict(PARAMS, bottom_level=1, prolong_form=form))
        got = []
        for fill in (False, True):
            if fill:
                S.set_ib_frac_compact(np.ones_like(p.vol), [np.ones_like(a) for a in p.area])
            S.set_zero_sol()
            info = S.cg_solve()
            assert info["status"] == 0, info
            got.append((S.launch_counts()[1], info["iterations"], S.get_sol_compact()))
        out.append(got)
    (a, b), (c, d) = out
    assert a[0] < b[0] < d[0] and a[0] < c[0]
    for x, y in ((a, c), (b, d)):
        assert x[1] == y[1]
        assert np.array_equal(x[2], y[2])


@pytest.mark.parametrize("name", ["config2", "c1"])
def test_launch_variants_of_separate_sweeps(name):
    if name == "c1":
        g, t, tb, S = setup_solver(name)
        S.set_rhs_compact(g["sv_rhs"])
    else:
        S = W.make_solver(W.config2())
    out = []
    for v in (3, 11, 12, 13):
        S.set_zero_sol()
        S.set_params(**dict(PARAMS, prolong_form=0, smooth_variant=v))
        info = S.cg_solve()
        assert info["status"] == 0, info
        out.append((info["iterations"], S.get_sol_compact()))
    for k in (1, 2, 3):
        assert out[0][0] == out[k][0], k
        assert np.array_equal(out[0][1], out[k][1]), k
