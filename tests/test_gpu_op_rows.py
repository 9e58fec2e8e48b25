"""The operator by rows that an FP32 solve applies by default (threads of four
cells of a row, exact FP32 differences where a block has one coefficient) against
the reference-order FP64 operator on the same FP32 values: rounding level, cell by
cell, for every block side it takes, all face kinds, cut cells, variable and
constant coefficients, a Helmholtz term, the lists of a forest and the reduced
ones, and values whose FP32 sums overflow or are denormal.  Where a block has one
coefficient, two roundings of the exact result."""
from fractions import Fraction

import numpy as np
import pytest

from sayakaamr_gb300 import workloads as W
from test_exact_delta import VALUES
from test_gpu_active import _tube
from test_gpu_async import _disk
from test_gpu_hybrid_f32 import _problem

pytestmark = pytest.mark.gpu

# a cell's sums have at most 2 ND + 4 terms a side in 3D (a refined face: four
# fine cells), each with up to four roundings of its coefficient and one of the
# product and the sum, in either operator
ROUNDINGS = 2 * 60 * 2.0 ** -53


def _scale(p, alpha, x):
    """a bound of |diag| |x| + sum |T x| per cell: B and the fractions up to 1.4, a
    face at a refined neighbour 4/3, at a wall 2, every |x| the largest, over vf"""
    h = p.tables["block_len"].reshape(-1, 3)[:, 0] / p.tables["nb"]
    b = max(np.abs(q).max() for q in p.bface)
    with np.errstate(over="ignore"):
        row = 2 * (2 * p.tables["ndim"] * 2 * b / h ** 2 + alpha)
    return np.repeat(row, p.ncell) / np.where(p.vol > 0, p.vol, 1.0).reshape(-1) * np.abs(x).max()


def _check(p, x, alpha=0.0, **kw):
    S = W.make_solver(p, use_mg_precond=1, bottom=1, precision=1, **kw)
    S.set_scalars(alpha, 1.0)
    x = x.astype(np.float32).astype(np.float64)
    y = S.device_apply_rows(x).reshape(p.num_blocks, -1)[p.leaf]
    ref = S.apply(int(p.tables["level"].max()), x).reshape(p.num_blocks, -1)[p.leaf]
    scale = _scale(p, alpha, x).reshape(p.num_blocks, -1)[p.leaf]
    assert np.isfinite(y).all() and np.abs(ref).max() > 0
    worst = (np.abs(y - ref) / scale).max()
    assert worst <= ROUNDINGS, worst
    return S


def _values(p, kind, seed=2):
    g = np.random.default_rng(seed)
    n = p.num_blocks * p.ncell
    if kind == "overflow":  # neighbours whose FP32 sums leave the range
        return g.choice([-3e38, 3e38, 1.0], n)
    if kind == "denormal":
        return g.standard_normal(n) * 1e-40
    return VALUES[kind](g, n)


@pytest.mark.parametrize("kind", list(VALUES) + ["overflow", "denormal"])
@pytest.mark.parametrize("nd, nb", [(2, 4), (2, 8), (2, 12), (2, 16), (3, 4), (3, 8), (3, 12), (3, 16)])
def test_against_the_reference_order(nd, nb, kind):
    p = _problem(nd, nb, 0.2)
    assert len(set(p.tables["level"][p.leaf])) > 1
    S = _check(p, _values(p, kind))
    assert S.uniform_blocks() > 0
    _check(p, _values(p, kind), uniform=0)
    if kind == "rough":
        _check(p, _values(p, kind), alpha=2.5)


@pytest.mark.parametrize("per_problem", [0, 1])
def test_forest(per_problem):
    p = W.forest([W.batch_problem(np.random.default_rng(k), "p%d" % k) for k in range(3)], "f")
    _check(p, _values(p, "rough"), per_problem=per_problem)


@pytest.mark.parametrize("problem", [lambda: _disk(3), lambda: _tube(0.06)], ids=["2d", "3d"])
def test_reduced_lists(problem):
    p = problem()
    S = _check(p, _values(p, "rough"))
    assert S.launch_counts()[0] == 4  # the lists are reduced


@pytest.mark.parametrize("kind", VALUES)
@pytest.mark.parametrize("nd, nb", [(2, 16), (3, 8)])
def test_two_roundings_where_a_block_has_one_coefficient(nd, nb, kind):
    p = _problem(nd, nb, 0.0)
    p.vol[:] = 1.0
    for d in range(nd):
        p.area[d][:] = 1.0
        p.bface[d][:] = 0.7
    S = W.make_solver(p, use_mg_precond=1, bottom=1, precision=1)
    x = _values(p, kind).astype(np.float32)
    y = S.device_apply_rows(x.astype(np.float64)).reshape((-1,) + (nb,) * nd)
    xb = x.reshape(y.shape)
    g = np.random.default_rng(1)
    h = p.tables["block_len"].reshape(-1, 3)[:, 0] / nb
    # (four cells of a row at a coarse/fine face take the general form)
    n, child = p.tables["neighbor"].reshape(-1, 6)[:, :2 * nd], p.tables["child"].reshape(-1, 8)[:, 0]
    inside = [b for b in p.leaf if (n[b] != -1).all() and (child[n[b][n[b] >= 0]] < 0).all()]
    assert len(inside) > 4
    for b in g.choice(inside, 40):
        T, S1 = (1.0 * h[b] ** (nd - 1)) / h[b] * 0.7, 1.0 / h[b] ** nd
        for _ in range(25):
            c = tuple(g.integers(1, nb - 1, nd))
            v = [xb[b][c[:q] + (c[q] + s,) + c[q + 1:]] for q in range(nd) for s in (-1, 1)]
            delta = 2 * nd * Fraction(float(xb[b][c])) - sum(Fraction(float(q)) for q in v)
            exact, top = Fraction(T * S1) * delta, max(abs(float(q)) for q in v + [xb[b][c]])
            bound = abs(exact) * (Fraction(2) ** -52 + Fraction(2) ** -100) + Fraction(T * S1 * top) * Fraction(2) ** -69
            assert abs(Fraction(float(y[b][c])) - exact) <= bound, (b, c)
