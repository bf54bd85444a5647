"""Blocks whose ranks outgrow their first workspace several times continue in the
growth arena: a build takes as many launches as one whose workspace holds every
rank from the start (a block that found the arena full would be compressed
again, in further launches), with the same factors' product."""
import numpy as np
import pytest

from hodlrnd_gb300 import _lib
from hodlrnd_gb300.kernels import Kernel
from hodlrnd_gb300.matrix import HODLRdD_matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ndim,n,dprime,eps,nmax", [(3, 8000, 2, 1e-10, 64), (2, 20000, 1, 1e-12, 64),
                                                    (4, 6000, 3, 1e-8, 128), (3, 3000, 0, 1e-12, 64)])
def test_blocks_grow_in_one_pass(ndim, n, dprime, eps, nmax):
    rng = np.random.default_rng(n + ndim)
    pts = rng.uniform(0.0, 1.0, (n, ndim))
    x = rng.standard_normal(n)

    def build(rank_cap):
        M = HODLRdD_matrix(Kernel("inv_r", 1.0 / n, 1.0), pts, [0.0] * ndim, [1.0] * ndim, Nmax=nmax, eps_ACA=eps,
                           INTERACTION_TYPE_ALLOWED=dprime, rank_cap=rank_cap)
        before = _lib.lib().hodlr_kernel_launches()
        M.Assemble_matrix_operators()
        return M, _lib.lib().hodlr_kernel_launches() - before

    M, launches = build(16)  # three growths for the highest ranks
    R, least = build(1024)
    assert int(M.blocks()["rank"].max()) > 4 * 16
    assert np.array_equal(M.blocks()["rank"], R.blocks()["rank"])
    assert launches == least
    assert np.array_equal(M * x, R * x)
    M.close()
    R.close()
