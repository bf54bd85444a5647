"""The CGS2 Arnoldi step sums its CTAs' shares with FP64's range: operators whose
|w|^2 passes FP32's 3.4e38 though no CTA's share of it does (n = 20011, a
152nd of the vector each) are solved."""
import numpy as np
import pytest

from hodlrnd_gb300.kernels import Kernel
from hodlrnd_gb300.matrix import HODLRdD_matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exponent", [62, 64, 65, 66])
def test_norms_beyond_fp32(exponent):
    n, scale = 20011, 2.0 ** exponent
    rng = np.random.default_rng(n)
    pts = rng.uniform(-1.0, 1.0, (n, 2))
    M = HODLRdD_matrix(Kernel("inv_r", scale / n, scale), pts, [-1.0] * 2, [1.0] * 2, Nmax=64, eps_ACA=1e-8, tol=1e-8,
                       precision="mixed", ortho="cgs2").Assemble_matrix_operators()
    M.solve(scale * rng.standard_normal(n))
    assert M.last_solve["converged"] == 1
    M.close()
