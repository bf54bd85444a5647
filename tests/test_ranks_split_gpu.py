"""Small operators' compression against the CPU oracle: every block's rank, and with
the ranks equal the product within 1e-12 (the order of FP64 sums), without
exception (test_work_split_gpu.py allows 1e-9 where a rank differs)."""
import numpy as np
import pytest

from hodlrnd_gb300.kernels import Kernel
from hodlrnd_gb300.matrix import HODLRdD_matrix
from oracle.oracle import OracleHODLR

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ndim,n,nmax", [(1, 3000, 20), (2, 33, 64), (2, 300, 33), (2, 2500, 100), (2, 9001, 64),
                                         (3, 1501, 8), (3, 5003, 48), (4, 2100, 128)])
def test_ranks_and_products_equal_the_oracles(ndim, n, nmax):
    rng = np.random.default_rng(100 * ndim + n)
    pts = rng.uniform(0.0, 1.0, (n, ndim))
    x = rng.uniform(0.5, 1.0, n)
    box = ([0.0] * ndim, [1.0] * ndim)
    O = OracleHODLR(pts, *box, nmax=nmax, dprime=0, eps=1e-9, kind=1, scale=1.0 / n, diag=1.0, rng_mode=1)
    M = HODLRdD_matrix(Kernel("inv_r", 1.0 / n, 1.0), pts, *box, Nmax=nmax, eps_ACA=1e-9).Assemble_matrix_operators()
    assert np.array_equal(M.blocks()["rank"], O.blocks()["rank"])
    yo = O.matvec(x)
    assert np.linalg.norm(M * x - yo) <= 1e-12 * np.linalg.norm(yo)
    M.close()
