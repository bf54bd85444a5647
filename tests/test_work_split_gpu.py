"""Products of small operators, whose phases are cut into short items with
many partial sums (item_bytes in engine.cu): sizes around one leaf, a few
parts and more than eight parts per sum, ragged leaves below, at and above 32
rows, against the CPU oracle's HODLR product.

FP64: both sides sum the same stored blocks (identical ranks), so they differ
by the order of FP64 sums only, 1e-12 as elsewhere.  FP32 factors: rounding
each factor entry to FP32 (2^-24) moves the product by at most
2 * 2^-24 * sum |U||V||x| -- for these positive kernels and vectors of one
sign the sums have no cancellation to speak of, so 1e-6 is a wide bound."""
import numpy as np
import pytest

from hodlrnd_gb300.kernels import Kernel
from hodlrnd_gb300.matrix import HODLRdD_matrix
from oracle.oracle import OracleHODLR

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("ndim,n,nmax", [(1, 3000, 20), (2, 33, 64), (2, 300, 33), (2, 2500, 100), (2, 9001, 64),
                                         (3, 1501, 8), (3, 5003, 48), (4, 2100, 128)])
def test_small_operator_products(ndim, n, nmax):
    rng = np.random.default_rng(100 * ndim + n)
    pts = rng.uniform(0.0, 1.0, (n, ndim))
    x = rng.uniform(0.5, 1.0, n)
    box = ([0.0] * ndim, [1.0] * ndim)
    k = Kernel("inv_r", 1.0 / n, 1.0)
    O = OracleHODLR(pts, *box, nmax=nmax, dprime=0, eps=1e-9, kind=1, scale=1.0 / n, diag=1.0, rng_mode=1)
    yo = O.matvec(x)
    M = HODLRdD_matrix(k, pts, *box, Nmax=nmax, eps_ACA=1e-9).Assemble_matrix_operators()
    y = M * x
    same = np.array_equal(M.blocks()["rank"], O.blocks()["rank"])
    assert rel(y, yo) <= (1e-12 if same else 1e-9)
    assert np.array_equal(M * x, y)  # partial sums in a fixed order
    M.close()
    M32 = HODLRdD_matrix(k, pts, *box, Nmax=nmax, eps_ACA=1e-9, precision="fp32_factors",
                         fp64_check=False).Assemble_matrix_operators()
    y32 = M32 * x
    assert rel(y32, yo) <= 1e-6
    assert np.array_equal(M32 * x, y32)
    M32.close()
