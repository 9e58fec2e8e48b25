"""Device memory that a solve can do without (the reduced block lists, the edge
words of the one-launch smoothing): a solve that cannot have it takes the full
lists and the separate launches and converges, and takes the faster route again
once the memory is there; a domain without solid blocks allocates no lists."""
import ctypes as C
import gc

import numpy as np
import pytest

from sayakaamr_gb300 import workloads as W
from test_gpu_active import _tube
from test_gpu_async import _disk

pytestmark = pytest.mark.gpu

PARAMS = dict(tol_rel=1e-10, tol_abs=0.0, use_mg_precond=1, bottom=1, precision=1, max_iter=500)


def _solve(S, p):
    S.set_zero_sol()
    info = S.cg_solve()
    assert info["status"] == 0, info
    r = S.residual(int(p.tables["level"].max()), S.get_sol_compact(), p.rhs).reshape(p.num_blocks, -1)[p.leaf]
    assert np.abs(r).max() < 2e-10 * info["rnorm0"]
    return S.launch_counts()[1]


@pytest.mark.parametrize("problem", [lambda: _disk(3), lambda: _tube(0.06)], ids=["2d", "3d"])
def test_solve_without_it(problem):
    p = problem()
    S, T = W.make_solver(p, **PARAMS), W.make_solver(p, **PARAMS)
    S.deny_optional_memory()
    without, usual = _solve(S, p), _solve(T, p)
    assert without > usual
    a, b = S.get_sol_compact(), T.get_sol_compact()
    assert np.linalg.norm(a - b) < 1e-7 * np.linalg.norm(b)
    S.deny_optional_memory(False)
    S.set_ib_frac_compact(p.vol, p.area)
    assert _solve(S, p) == usual
    assert np.array_equal(S.get_sol_compact(), b)


def _pool_used():
    cu = C.CDLL("libcuda.so.1")
    pool, used = C.c_void_p(), C.c_uint64()
    assert cu.cuDeviceGetDefaultMemPool(C.byref(pool), 0) == 0
    assert cu.cuMemPoolGetAttribute(pool, 7, C.byref(used)) == 0  # CU_MEMPOOL_ATTR_USED_MEM_CURRENT
    return used.value


def test_no_lists_without_solid_blocks():
    # blocks of 10 cells: no one-launch smoothing either
    p = W.config3(nb=10, max_level=4, band=1.0)
    p.vol[:] = 1.0
    for a in p.area:
        a[:] = 1.0
    used = []
    for deny in (True, False):
        S = W.make_solver(p, **PARAMS)
        S.deny_optional_memory(deny)
        gc.collect()
        base = _pool_used()
        S.prepare()
        used.append(_pool_used() - base)
        del S
    # the flags of the blocks; the lists would be 170 bytes for each entry of every list
    assert 0 <= used[1] - used[0] < 170 * p.num_blocks, used


@pytest.mark.parametrize("n, level", [(5, 1), (8, 2), (9, 2)])
def test_bottom_inverse_without_a_second_copy_of_all_matrices(n, level):
    # (8 and 9 matrices of order 1024: two copies of all do not fit the L2, and
    # two halves are inverted one after the other)
    p = W.forest([W.batch_problem(np.random.default_rng(k), "p%d" % k) for k in range(n)], "f")
    out = []
    for deny in (True, False):
        S = W.make_solver(p, **dict(PARAMS, tol_rel=1e-8, bottom_level=level))
        S.deny_optional_memory(deny)
        S.set_params(prolong_form=0)  # the edge words are not what is compared
        info = S.cg_solve()
        assert info["status"] == 0, info
        out.append((info["iterations"], S.get_sol_compact()))
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1], out[1][1])
