"""The restriction onto coarse blocks (two coarse cells per thread where the
blocks' sides are a multiple of four, one elsewhere) against the C oracle: the
same bits, with cut cells, solid cells and blocks without either."""
import numpy as np
import pytest

from sayakaamr_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nd,nb", [(2, 4), (2, 6), (2, 8), (2, 10), (2, 12), (2, 16), (3, 4), (3, 6), (3, 8), (3, 12)])
def test_restriction_matches_the_oracle(nd, nb):
    from oracle import pyoracle
    p = W.config2(nb=nb, max_level=4) if nd == 2 else W.config3(nb=nb, max_level=3, band=1.0)
    vf, af, bc = pyoracle.setup_coefficients(p.tables, p.bc, p.vol, p.area, p.bface)
    S = W.make_solver(p)
    x = np.random.default_rng(nb).standard_normal(S.num_blocks * S.ncell)
    ref = pyoracle.Oracle(p.tables, p.bc, vf, af, bc).restrict_sweep(x)
    assert np.array_equal(S.restrict_sweep(x).view(np.int64), ref.view(np.int64))


@pytest.mark.parametrize("nd,precision", [(2, 0), (2, 1), (3, 0), (3, 1)])
def test_block_records_give_the_bits_of_the_arrays(nd, precision):
    p = W.config2(nb=8, max_level=5) if nd == 2 else W.config3(nb=8, max_level=4, band=1.0)
    out = []
    for uniform in (1, 0):
        S = W.make_solver(p, tol_rel=1e-9, tol_abs=0.0, use_mg_precond=1, bottom=1, precision=precision, max_iter=200,
                          uniform=uniform)
        info = S.cg_solve()
        out.append((info["status"], info["iterations"], info["rnorm"], S.get_sol_compact()))
    assert out[0][:3] == out[1][:3]
    assert np.array_equal(out[0][3], out[1][3])
