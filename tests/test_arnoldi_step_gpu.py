"""The one-launch Arnoldi step (vectors of up to 40960 points, restart up to
255) against the separate orthogonalisation kernels: the same Krylov space, so
the same iteration count up to a residual that falls on the tolerance itself
(+-1) and solutions that differ by the solver tolerance times the conditioning
(well below 10 here: the operators are the identity plus a small integral
operator).  Sizes: a few points (most CTAs of the cluster without any), one
element per thread, several, and either side of the limit; with restarts."""
import numpy as np
import pytest

from hodlrnd_gb300.kernels import Kernel
from hodlrnd_gb300.matrix import HODLRdD_matrix

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("n,precision,ortho", [(3, "fp64", "mgs"), (70, "fp64", "cgs2"), (2111, "fp64", "mgs"),
                                               (2111, "mixed", "mgs"), (2111, "mixed", "cgs2"),
                                               (20011, "fp32_factors", "cgs2"), (20011, "fp64", "mgs"),
                                               (40960, "fp32_factors", "cgs2"), (40960, "fp64", "mgs"),
                                               (40961, "fp64", "mgs")])
def test_step_matches_separate_kernels(n, precision, ortho):
    rng = np.random.default_rng(n)
    pts = rng.uniform(-1.0, 1.0, (n, 2))
    b = rng.standard_normal(n)
    M = HODLRdD_matrix(Kernel("inv_r", 1.0 / n, 1.0), pts, [-1.0] * 2, [1.0] * 2, Nmax=64, eps_ACA=1e-8, tol=1e-8,
                       precision=precision, ortho=ortho).Assemble_matrix_operators()
    x = M.solve(b)
    a = dict(M.last_solve)
    assert a["converged"] == 1
    assert np.array_equal(M.solve(b), x)
    M.set_solver(restart=300, tol=1e-8)  # more basis vectors than a step takes: separate kernels
    y = M.solve(b)
    c = dict(M.last_solve)
    assert c["converged"] == 1
    assert abs(a["iterations"] - c["iterations"]) <= a["outer_iterations"] + c["outer_iterations"]
    assert rel(x, y) <= 2e-7
    M.set_solver(restart=4, tol=1e-8, max_iter=5000)  # GMRES(4) needs 307 iterations at n = 70
    z = M.solve(b)
    assert M.last_solve["converged"] == 1
    assert rel(z, y) <= 2e-7
    M.close()
