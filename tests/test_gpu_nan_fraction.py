"""A volume fraction that is a NaN counts as solid, as every `vf > 0` takes it:
a solve over full block lists with such a cell inside a body gives the solution
of the same cell with fraction 0."""
import numpy as np
import pytest

from sayakaamr_gb300 import workloads as W
from test_gpu_async import _disk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_nan_inside_a_body(precision):
    # (one state per problem: no reduced lists; the disk lies in the upper
    # quadrants, so the cell's ancestors are solid up to the coarsest level)
    p = W.forest([_disk(3), _disk(4)], "disks")
    c = W.cell_centres(p.tables).reshape(p.num_blocks, p.ncell, -1)
    leaf = np.zeros(p.num_blocks, bool)
    leaf[p.leaf] = True
    b = np.nonzero(leaf & (np.abs(c[:, 0, :2] - [0.8, 0.2]).max(axis=1) < 0.1))[0][0]
    out = []
    for v in (0.0, np.nan):
        vol = p.vol.copy().reshape(p.num_blocks, -1)
        assert vol[b].max() == 0
        vol[b, 5] = v
        S = W.make_solver(p, tol_rel=1e-8, tol_abs=0.0, use_mg_precond=1, bottom=1, max_iter=200, precision=precision)
        S.set_ib_frac_compact(vol.reshape(-1), p.area)
        info = S.cg_solve()
        out.append((info["status"], info["iterations"], S.get_sol_compact()))
    assert out[0][0] == 0 and out[0][:2] == out[1][:2]
    assert np.array_equal(out[0][2], out[1][2])
