"""A solver workspace is complete when the call that allocates it returns, whatever
is queued on the default stream: a solve on another stream right after it has the
bits of one on an idle device (its clearing once waited on the default stream
behind the caller's work, and then ran into the solve)."""
import numpy as np
import pytest

from hodlrnd_gb300.kernels import Kernel
from hodlrnd_gb300.matrix import HODLRdD_matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,ortho", [("fp64", "mgs"), ("fp64", "cgs2"), ("mixed", "cgs2")])
def test_solve_right_after_a_larger_workspace(precision, ortho):
    torch = pytest.importorskip("torch")
    n = 2111
    rng = np.random.default_rng(n)
    pts = rng.uniform(-1.0, 1.0, (n, 2))
    b = rng.standard_normal(n)
    M = HODLRdD_matrix(Kernel("inv_r", 1.0 / n, 1.0), pts, [-1.0] * 2, [1.0] * 2, Nmax=64, eps_ACA=1e-8, tol=1e-8,
                       precision=precision, ortho=ortho).Assemble_matrix_operators()
    x = M.solve(b)
    a = torch.randn((4096, 4096), device="cuda")
    for restart in (120, 140, 160):
        torch.cuda.synchronize()
        for _ in range(100):  # tens of milliseconds on the default stream
            a = a @ a
            a = a / a.norm()
        M.set_solver(restart=restart, tol=1e-8)
        assert np.array_equal(M.solve(b), x)
    M.close()
