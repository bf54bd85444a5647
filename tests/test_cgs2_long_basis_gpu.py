"""CGS2 steps whose basis is too long for shared memory (more than 56 vectors at
n = 40,960, 73 at 30,000) read it from memory: a badly conditioned operator that
takes well over a hundred iterations, in the step kernels (restart 200) against the
separate kernels (restart 300), and the same bits when done phase by phase."""
import ctypes

import numpy as np
import pytest

from hodlrnd_gb300 import _lib
from hodlrnd_gb300.kernels import Kernel
from hodlrnd_gb300.matrix import HODLRdD_matrix

pytestmark = pytest.mark.gpu
STEP_WAIT_NS, STEPS = 3, 0


@pytest.mark.parametrize("n,precision", [(30000, "fp64"), (40960, "fp32_factors"), (40960, "mixed")])
def test_basis_beyond_shared_memory(n, precision):
    rng = np.random.default_rng(n)
    pts = rng.uniform(0.0, 1.0, (n, 3))
    b = rng.standard_normal(n)
    # a diagonal inside the integral operator's spectrum: slow convergence
    M = HODLRdD_matrix(Kernel("inv_r", n ** (-2.0 / 3.0), 0.6), pts, [0.0] * 3, [1.0] * 3, Nmax=64, eps_ACA=1e-8, tol=1e-8,
                       precision=precision, ortho="cgs2", fp64_check=False).Assemble_matrix_operators()

    def solve(restart):
        M.set_solver(restart=restart, tol=1e-8, max_iter=2000, inner_tol=1e-5)
        v0, v1 = ctypes.c_int64(), ctypes.c_int64()
        _lib.check(_lib.lib().hodlr_test_value(M._op, STEPS, ctypes.byref(v0)))
        x = M.solve(b)
        _lib.check(_lib.lib().hodlr_test_value(M._op, STEPS, ctypes.byref(v1)))
        return x, dict(M.last_solve), v1.value - v0.value

    x, info, steps = solve(200)
    assert info["converged"] == 1 and steps >= 90
    y, sep, none = solve(300)
    assert sep["converged"] == 1 and none == 0
    assert np.linalg.norm(x - y) <= 1e-5 * np.linalg.norm(y)
    _lib.check(_lib.lib().hodlr_test_option(M._op, STEP_WAIT_NS, 0))
    z, again, steps2 = solve(200)
    assert np.array_equal(x, z) and again["iterations"] == info["iterations"] and steps2 == steps
    M.close()
