"""A one-launch CGS2 step whose CTAs do not all get onto the device in time (its
wait is set to nothing here, so that it runs out at most barriers) is done again
phase by phase: the solve converges as without, with the same bits, in FP64 and
FP32, with the basis in shared memory and beyond it, over restarts."""
import ctypes

import numpy as np
import pytest

from hodlrnd_gb300 import _lib
from hodlrnd_gb300.kernels import Kernel
from hodlrnd_gb300.matrix import HODLRdD_matrix

pytestmark = pytest.mark.gpu
STEP_WAIT_NS, STEPS, GIVE_UPS = 3, 0, 1


def value(M, what):
    v = ctypes.c_int64()
    _lib.check(_lib.lib().hodlr_test_value(M._op, what, ctypes.byref(v)))
    return v.value


@pytest.mark.parametrize("n,precision,restart", [(40, "fp64", 3), (2111, "fp64", 100), (2111, "mixed", 5),
                                                 (20011, "fp32_factors", 100), (40960, "fp64", 4)])
def test_same_bits_when_the_device_is_busy(n, precision, restart):
    rng = np.random.default_rng(n)
    pts = rng.uniform(-1.0, 1.0, (n, 2))
    b = rng.standard_normal(n)
    M = HODLRdD_matrix(Kernel("inv_r", 1.0 / n, 1.0), pts, [-1.0] * 2, [1.0] * 2, Nmax=64, eps_ACA=1e-8, tol=1e-8,
                       precision=precision, ortho="cgs2").Assemble_matrix_operators()
    M.set_solver(restart=restart, tol=1e-8, max_iter=5000)
    x = M.solve(b)
    info, steps = dict(M.last_solve), value(M, STEPS)
    assert info["converged"] == 1 and steps == info["iterations"] > 0 and value(M, GIVE_UPS) == 0
    _lib.check(_lib.lib().hodlr_test_option(M._op, STEP_WAIT_NS, 0))
    y = M.solve(b)
    assert value(M, GIVE_UPS) > 0
    assert M.last_solve["iterations"] == info["iterations"] and M.last_solve["converged"] == 1
    assert np.array_equal(x, y)
    _lib.check(_lib.lib().hodlr_test_option(M._op, STEP_WAIT_NS, -1))
    gave = value(M, GIVE_UPS)
    assert np.array_equal(M.solve(b), x) and value(M, GIVE_UPS) == gave
    M.close()
