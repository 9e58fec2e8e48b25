"""Solvers used by several threads at once, each on its own stream: the one-launch
smoothing of a solver holds the device's blocks to itself, and solves that run
beside each other give the bits of solves that run alone."""
import threading

import numpy as np
import pytest

from sayakaamr_gb300 import workloads as W
from test_gpu_active import _tube
from test_gpu_async import _disk

pytestmark = pytest.mark.gpu

PARAMS = dict(tol_rel=1e-8, tol_abs=0.0, use_mg_precond=1, bottom=1, precision=1, max_iter=300)


def test_solves_beside_each_other():
    problems = [W.config2(nb=16, max_level=5), W.config2(nb=8, max_level=5), _tube(5.0), _disk(3)]
    solvers = [W.make_solver(p, **PARAMS) for p in problems]

    def solve(S):
        S.set_zero_sol()
        info = S.cg_solve()
        return info["status"], info["iterations"], S.get_sol_compact()

    alone = [solve(S) for S in solvers]
    assert all(a[0] == 0 for a in alone)
    wrong = []

    def work(k):
        for _ in range(12):
            try:
                r = solve(solvers[k])
            except Exception as e:  # reported below, in the main thread
                wrong.append((k, e))
                return
            if r[:2] != alone[k][:2] or not np.array_equal(r[2], alone[k][2]):
                wrong.append((k, r[:2]))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(solvers))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong
