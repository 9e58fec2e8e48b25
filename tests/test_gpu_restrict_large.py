"""The restriction on levels large enough for two coarse cells per thread (131,072
cells and more), and on those just below, against the C oracle: the same bits."""
import numpy as np
import pytest

from sayakaamr_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _cells(p, level):
    tb = p.tables
    return int(((tb["level"] == level) & (tb["node_type"] != 1)).sum()) * p.ncell


@pytest.mark.parametrize("problem", [lambda: W.config2(nb=16, max_level=8), lambda: W.config3(nb=8, max_level=5),
                                     lambda: W.config3(nb=12, max_level=5)], ids=["2d-16", "3d-8", "3d-12"])
def test_restriction_matches_the_oracle(problem):
    from oracle import pyoracle
    p = problem()
    sizes = [_cells(p, l) for l in range(1, int(p.tables["level"].max()))]
    assert min(sizes) < 1 << 17 <= max(sizes), sizes
    vf, af, bc = pyoracle.setup_coefficients(p.tables, p.bc, p.vol, p.area, p.bface)
    S = W.make_solver(p)
    x = np.random.default_rng(3).standard_normal(S.num_blocks * S.ncell)
    ref = pyoracle.Oracle(p.tables, p.bc, vf, af, bc).restrict_sweep(x)
    assert np.array_equal(S.restrict_sweep(x).view(np.int64), ref.view(np.int64))
