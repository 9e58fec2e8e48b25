"""The launches that a solve reports before its iterations: x0 and the first
residual, one more for the states of a forest, one (FP64) or two (FP32) more for
the zeros of the solid blocks where the reduced lists are walked."""
import pytest

from sayakaamr_gb300 import workloads as W
from test_gpu_async import _disk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("problem, precision, launches",
                         [(lambda: W.config2(nb=8, max_level=3), 1, 2),
                          (lambda: W.forest([_disk(3), _disk(4)], "disks"), 1, 3),
                          (lambda: _disk(3), 1, 4), (lambda: _disk(3), 0, 3)],
                         ids=["plain", "forest", "solid-fp32", "solid-fp64"])
def test_prologue(problem, precision, launches):
    S = W.make_solver(problem(), use_mg_precond=1, bottom=1, precision=precision)
    S.prepare()
    assert S.launch_counts()[0] == launches
