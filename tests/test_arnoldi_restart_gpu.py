"""Which Arnoldi kernels a solve takes depends on that solve's restart alone: a
short cycle takes the one-launch step on an operator that has had a long one (255
basis vectors and more take the separate kernels), with the bits of an operator
that has not; its restarts go through the step kernels."""
import ctypes

import numpy as np
import pytest

from hodlrnd_gb300 import _lib
from hodlrnd_gb300.kernels import Kernel
from hodlrnd_gb300.matrix import HODLRdD_matrix

pytestmark = pytest.mark.gpu
STEPS = 0


def steps(M):
    v = ctypes.c_int64()
    _lib.check(_lib.lib().hodlr_test_value(M._op, STEPS, ctypes.byref(v)))
    return v.value


@pytest.mark.parametrize("n,precision,ortho,restart", [(2111, "fp64", "mgs", 4), (2111, "fp64", "cgs2", 5),
                                                       (2111, "mixed", "mgs", 3), (5000, "fp32_factors", "cgs2", 255),
                                                       (5000, "bf16_factors", "cgs2", 4), (70, "fp64", "mgs", 254)])
def test_a_long_cycle_leaves_nothing_behind(n, precision, ortho, restart):
    rng = np.random.default_rng(n)
    pts = rng.uniform(-1.0, 1.0, (n, 2))
    b = rng.standard_normal(n)
    M = HODLRdD_matrix(Kernel("inv_r", 1.0 / n, 1.0), pts, [-1.0] * 2, [1.0] * 2, Nmax=64, eps_ACA=1e-8, tol=1e-8,
                       precision=precision, ortho=ortho).Assemble_matrix_operators()

    def solve(r):
        M.set_solver(restart=r, tol=1e-8, max_iter=5000)
        before = steps(M)
        x = M.solve(b)
        assert M.last_solve["converged"] == 1
        return x, M.last_solve["iterations"], steps(M) - before

    x, its, taken = solve(restart)
    assert its > 0 and taken >= its - M.last_solve["outer_iterations"]
    z, its300, taken300 = solve(300)
    assert its300 > 0 and taken300 == 0
    assert np.linalg.norm(z - x) <= 2e-7 * np.linalg.norm(x)
    y, its2, taken2 = solve(restart)
    assert (its2, taken2) == (its, taken) and np.array_equal(x, y)
    M.close()
