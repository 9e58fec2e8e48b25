"""The smoothing of a tower in one cooperative launch (FP32; 2D blocks of 8 or
16 cells, 3D blocks of 8; prolong_form 1) against the separate
launches (prolong_form 0): the same bits, on trees of one block per problem up
to more blocks than a launch can hold, with coarse/fine and physical faces,
cut cells, solid blocks (reduced lists), over-relaxation, one to five sweeps,
and a forest whose problems finish at different iterations."""
import numpy as np
import pytest

from sayakaamr_gb300 import workloads as W

pytestmark = pytest.mark.gpu

PARAMS = dict(tol_rel=1e-10, tol_abs=0.0, use_mg_precond=1, bottom=1, precision=1, max_iter=500)


def _both(p, **kw):
    out = []
    for form in (1, 0):
        S = W.make_solver(p, **dict(PARAMS, prolong_form=form, **kw))
        for _ in range(2):  # the second solve runs on the first one's words
            S.set_zero_sol()
            info = S.cg_solve()
        # (whether 1e-10 is within reach of a tree's true residual or not, the
        # solves take the same steps)
        out.append((info["status"], info["iterations"], info["rnorm"], S.get_sol_compact()))
    assert out[0][:3] == out[1][:3]
    assert np.array_equal(out[0][3], out[1][3])


@pytest.mark.parametrize("nb", [8, 16])
@pytest.mark.parametrize("levels", [2, 4, 6])
@pytest.mark.parametrize("kw", [dict(), dict(relax_omega=1.1, n_post_smooth=3), dict(n_post_smooth=1),
                                dict(n_post_smooth=5, uniform=0)], ids=["2", "3-relaxed", "1", "5-arrays"])
def test_same_bits_as_the_separate_launches(nb, levels, kw):
    _both(W.config2(nb=nb, max_level=levels), **kw)


def test_many_blocks_and_mixed_towers():
    # the coarse towers fit a launch, the finest one does not
    _both(W.config2(nb=8, max_level=8))


@pytest.mark.parametrize("n", [2, 9])
def test_forest(n):
    _both(W.forest([W.batch_problem(np.random.default_rng(k), "p%d" % k) for k in range(n)], "f"), relax_omega=1.1,
          tol_rel=1e-8)


@pytest.mark.parametrize("nb", [8, 16])
def test_mostly_solid(nb):
    # fluid inside a disk only: more than a quarter of the blocks is solid
    t = W.refine_tree(2, nb, (2, 2, 1), (0, 0, 0), (1, 1, 0), 3, 6,
                      lambda lo, hi, l: np.abs(np.hypot(*(0.5 * (lo + hi) - [0.45, 0.8]).T) - 0.2) < 1.2 * (hi - lo)[:, 0])
    tb = t.tables()
    d = lambda p: 0.2 - np.hypot(p[..., 0] - 0.45, p[..., 1] - 0.82)  # noqa: E731
    vol = (d(W.cell_centres(tb)) > 0).astype(np.float64)
    area = [(d(W.face_centres(tb, q)) > 0).astype(np.float64) for q in range(2)]
    f = W.gaussian_rhs(np.random.default_rng(3), W.cell_centres(tb), 2)
    p = W._finish("disk", t, tb, vol, area, [np.ones_like(a) for a in area], f, False, {}, dirichlet_faces=(3,))
    assert 4 * (p.vol.reshape(p.num_blocks, -1).max(axis=1) == 0).sum() > p.num_blocks
    _both(p)


@pytest.mark.parametrize("levels", [2, 4, 5])
@pytest.mark.parametrize("kw", [dict(), dict(relax_omega=1.1, n_post_smooth=4), dict(n_post_smooth=1, uniform=0)],
                         ids=["2", "4-relaxed", "1-arrays"])
def test_3d(levels, kw):
    # at 5 levels the finest tower holds more blocks than a launch
    _both(W.config3(nb=8, max_level=levels, band=1.0), **kw)


@pytest.mark.parametrize("kw", [dict(n_post_smooth=4, relax_omega=1.1), dict(n_post_smooth=3)], ids=["4", "3"])
def test_3d_moving_body(kw):
    """mostly solid (reduced lists); the fractions change under a captured
    graph, by a little and by so much that other towers fit a launch"""
    seq = list(W.config5_sequence(steps=3, regrid_every=100, max_level=5))
    out = []
    for form in (1, 0):
        S = W.make_solver(seq[0][2], **dict(PARAMS, prolong_form=form, bottom_level=1, **kw))
        got = []
        for _, _, p in seq + seq[:1]:
            S.set_ib_frac_compact(p.vol, p.area)
            S.set_rhs_compact(p.rhs)
            S.set_zero_sol()
            info = S.cg_solve()
            got.append((info["status"], info["iterations"], S.get_sol_compact()))
        full = np.ones_like(p.vol)
        S.set_ib_frac_compact(full, [np.ones_like(a) for a in p.area])
        S.set_zero_sol()
        info = S.cg_solve()
        got.append((info["status"], info["iterations"], S.get_sol_compact()))
        out.append(got)
    for a, b in zip(*out):
        assert a[:2] == b[:2]
        assert np.array_equal(a[2], b[2])


@pytest.mark.parametrize("variant", [11, 12, 13])
@pytest.mark.parametrize("kw", [dict(), dict(relax_omega=1.1, n_post_smooth=3), dict(uniform=0)],
                         ids=["2", "3-relaxed", "arrays"])
def test_row_sweeps_of_3d_blocks(variant, kw):
    """3D blocks of 8^3 cells, one thread per row, in towers too large for one
    launch: the same bits as one thread per cell (variant 3)"""
    p = W.config3(nb=8)
    out = []
    for v, form in ((variant, 1), (3, 0)):
        S = W.make_solver(p, **dict(PARAMS, smooth_variant=v, prolong_form=form, **kw))
        info = S.cg_solve()
        out.append((info["status"], info["iterations"], info["rnorm"], S.get_sol_compact()))
    assert out[0][:3] == out[1][:3]
    assert np.array_equal(out[0][3], out[1][3])
