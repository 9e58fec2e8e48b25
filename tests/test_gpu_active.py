"""The device solve's block lists without the solid blocks: a domain that is
mostly body (the elbow pipe: more than a quarter of the blocks hold no fluid).
What the solid blocks of the work vectors and of the initial solution hold
does not reach the result, the solution keeps its given values there, and the
solution satisfies the reference-order operator.  Domains on both sides of
the switch: without a solid block, with a few, mostly solid."""
import numpy as np
import pytest

from sayakaamr_gb300 import workloads as W

pytestmark = pytest.mark.gpu

PARAMS = dict(tol_rel=1e-10, tol_abs=0.0, use_mg_precond=1, bottom=1, max_iter=500)


def _tube(radius, nb=8):
    """elbow tree at 4 levels, fluid within `radius` of the centreline"""
    t = W.elbow_tree(W.elbow_point(0.4), nb=nb, max_level=4)
    tb = t.tables()
    d = lambda p: radius - W.elbow_dist(p)  # noqa: E731
    vol = (d(W.cell_centres(tb)) > 0).astype(np.float64)
    area = [(d(W.face_centres(tb, q)) > 0).astype(np.float64) for q in range(3)]
    bface = [np.ones_like(a) for a in area]
    f = W.gaussian_rhs(np.random.default_rng(3), W.cell_centres(tb), 3, sigma=0.08)
    return W._finish("tube", t, tb, vol, area, bface, f, False, {}, dirichlet_faces=(0,))


@pytest.mark.parametrize("radius", [0.06, 0.1, 0.45, 5.0])
@pytest.mark.parametrize("params", [dict(precision=1), dict(precision=0), dict(precision=1, smoother=1, n_post_smooth=3),
                                    dict(precision=0, smoother=1, n_post_smooth=3),
                                    dict(precision=1, sublevel_order=0), dict(precision=1, vcycle_out=2)],
                         ids=lambda p: "-".join("%s%s" % kv for kv in p.items()))
def test_solid_blocks_do_not_matter(radius, params):
    p = _tube(radius)
    n, nc = p.num_blocks, p.ncell
    solid = ~(p.vol.reshape(n, nc) > 0).any(axis=1)
    x0 = np.zeros((n, nc))
    x0[solid] = np.random.default_rng(1).standard_normal((int(solid.sum()), nc))
    S = W.make_solver(p, **PARAMS, **params)
    S.set_init_sol(x0.reshape(-1))
    info = S.cg_solve()
    assert info["status"] == 0, info
    a = S.get_sol_compact().reshape(n, nc)
    leaf = p.tables["node_type"] == 1
    r = S.residual(int(p.tables["level"].max()), a.reshape(-1), p.rhs).reshape(n, nc)[leaf]
    assert np.abs(r).max() < 2e-10 * info["rnorm0"]
    assert np.array_equal(a[solid], x0[solid])
    # a solver whose work vectors hold other values everywhere, also in the
    # solid blocks, and which starts from zero there
    T = W.make_solver(p, **PARAMS, **params)
    T.cg_solve()
    junk = np.random.default_rng(2).standard_normal(n * nc)
    T.smooth(int(p.tables["level"].max()), junk, junk)
    T.device_smooth(int(p.tables["level"].max()), junk, junk, 3)
    T.device_apply(junk)
    T.set_zero_sol()
    again = T.cg_solve()
    b = T.get_sol_compact().reshape(n, nc)
    assert again["iterations"] == info["iterations"]
    assert np.array_equal(a[~solid], b[~solid])
