"""The FP32 block-hybrid pass as the V-cycle runs it (blocks in registers: one
warp per 16x16 block, one thread per row of an 8^3 or 16^3 block) against the
general kernel: the same bits, on towers with coarse/fine, Dirichlet and Neumann
faces, cut and solid cells, blocks with one coefficient and with many, the record
of the former on and off, and with the prolongation of the tower's own level done
by the pass instead of before it."""
import numpy as np
import pytest

from sayakaamr_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _problem(nd, nb, radius):
    """a refined spot in the unit box, B = 1 on one side of it; fluid outside a ball"""
    mid = np.array([0.55, 0.45, 0.5])[:nd]
    t = W.refine_tree(nd, nb, (2, 1, 1), (0, 0, 0), (2, 1, 1 if nd == 3 else 0), 2, 4,
                      lambda lo, hi, l: np.linalg.norm((0.5 * (lo + hi))[:, :nd] - mid, axis=1) < 0.9 * (hi - lo)[:, 0])
    tb = t.tables()
    d = lambda p: np.linalg.norm(p[..., :nd] - mid, axis=-1) - radius  # noqa: E731
    vol = (d(W.cell_centres(tb)) > 0).astype(np.float64)
    area, b = [], []
    for q in range(nd):
        x = W.face_centres(tb, q)
        area.append((d(x) > 0).astype(np.float64))
        b.append(np.where(x[..., 0] > 0.5, 1.0 + 0.4 * np.sin(9 * x[..., 0] + 5 * x[..., 1]), 1.0))
    f = W.gaussian_rhs(np.random.default_rng(1), W.cell_centres(tb), nd)
    return W._finish("spot", t, tb, vol, area, b, f, False, {}, dirichlet_faces=(1, 2))


def _same(S, tb, seed):
    g = np.random.default_rng(seed)
    n = S.num_blocks * S.ncell
    phi, rhs = g.standard_normal(n), g.standard_normal(n)
    finest = int(tb["level"].max())
    for L in (finest, finest - 1):
        for sweeps in (1, 2, 3):
            for prolong in (False, True):
                a = S.device_hybrid_pass_f32(L, phi, rhs, sweeps, prolong=prolong)
                b = S.device_hybrid_pass_f32(L, phi, rhs, sweeps, general=True, prolong=prolong)
                assert np.isfinite(a).all()
                assert not np.array_equal(a, phi.astype(np.float32).astype(np.float64))
                assert np.array_equal(a, b), (L, sweeps, prolong, np.flatnonzero(a != b)[:8])


@pytest.mark.parametrize("kw", [dict(), dict(uniform=0), dict(relax_omega=1.2)], ids=["records", "arrays", "relaxed"])
@pytest.mark.parametrize("radius", [0.0, 0.2])
@pytest.mark.parametrize("nd, nb", [(2, 16), (3, 8), (3, 16)])
def test_same_bits_as_the_general_kernel(nd, nb, radius, kw):
    p = _problem(nd, nb, radius)
    S = W.make_solver(p, use_mg_precond=1, bottom=1, precision=1, **kw)
    assert len(set(p.tables["level"][p.leaf])) > 1
    assert S.uniform_blocks() > 0
    _same(S, p.tables, nb)


def _pairs(q, nd, g):
    """(B, a) with a = 1 and a = 3/4 whose face coefficients (q B) a agree to the
    last bit, while the FP32 diagonals of a cell with its third face at a coarser
    neighbour do not"""
    f = np.float32

    def diagonal(b, a):
        t = f((q * b) * a)
        s = f(f(t + t) + f(f(f(f(q) / f(1.5)) * f(b)) * f(a)))
        for _ in range(2 * nd - 3):
            s = f(s + t)
        return s
    while True:
        b1 = 1.0 + g.random()
        for k in range(-3, 4):
            b2 = b1 / 0.75 + k * np.spacing(b1 / 0.75)
            if (q * b2) * 0.75 == q * b1 and diagonal(b1, 1.0) != diagonal(b2, 0.75):
                return (b1, 1.0), (b2, 0.75)


@pytest.mark.parametrize("nd, nb", [(2, 16), (3, 8), (3, 16)])
def test_coefficient_of_varying_factors(nd, nb):
    """B and the area fraction vary against each other and their product does
    not: one coefficient on every face of a block, but two on those at a coarser
    neighbour"""
    p = _problem(nd, nb, 0.0)
    tb = p.tables
    g = np.random.default_rng(5)
    fine = int(tb["level"].max())
    for d in range(nd):
        x = W.face_centres(tb, d)
        dx = tb["block_len"].reshape(-1, 3)[:, 0] / nb
        # beta ds / dx, a power of two as the spacings are (the factor's own bits do not matter)
        h = dx[tb["level"] == fine][0]
        (b1, a1), (b2, a2) = _pairs(h ** (nd - 1) / h, nd, g)
        assert len(np.unique(dx)) == fine
        step = np.round(2 * x / dx.reshape((-1,) + (1,) * (x.ndim - 1))).astype(np.int64)[..., :nd].sum(axis=-1) // 2
        p.bface[d][...] = np.where(step % 2 == 0, b1, b2).reshape(p.bface[d].shape)
        p.area[d][...] = np.where(step % 2 == 0, a1, a2).reshape(p.area[d].shape)
    S = W.make_solver(p, use_mg_precond=1, bottom=1, precision=1)
    assert S.uniform_blocks() > 0
    _same(S, tb, 3)
