"""How the FP32 V-cycle's output reaches the BiCGSTAB kernels by default
(vcycle_out 0) on 3D towers of more than 2,097,152 cells, by the launches of an
iteration (widening takes two more): in place where the operator by rows takes
the blocks (a side that is a multiple of four), widened where it does not."""
import pytest

from sayakaamr_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb, like", [(10, 2), (8, 3)])
def test_default_on_large_3d_towers(nb, like):
    p = W.config3(nb=nb, max_level=5 if nb == 10 else 6, band=3.0 if nb == 10 else 2.0)
    assert p.leaf.size * p.ncell > 1 << 21
    S = W.make_solver(p, use_mg_precond=1, bottom=1, precision=1)
    launches = {}
    for form in (0, 2, 3):
        S.set_params(vcycle_out=form)
        S.prepare()
        launches[form] = S.launch_counts()[1]
    assert launches[2] == launches[3] + 2
    assert launches[0] == launches[like], launches
