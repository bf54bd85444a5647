"""FP64 operators of very many tiny far segments, whose leaf panels take a kernel of
their own (half a million segments and more; 2.9 and about 1 rows a panel): products
against the CPU oracle, which sums the same stored blocks (1e-12, the order of FP64
sums), the same bits each time, and the same bits as a member of a batch beside an
operator that takes the other route."""
import numpy as np
import pytest

from hodlrnd_gb300.batch import HODLRdD_batch
from hodlrnd_gb300.kernels import Kernel
from hodlrnd_gb300.matrix import HODLRdD_matrix
from oracle.oracle import OracleHODLR

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ndim,n,nmax", [(5, 3000, 64), (4, 3000, 6)])
def test_products_of_tiny_segments(ndim, n, nmax):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(ndim * n)
    box = ([0.0] * ndim, [1.0] * ndim)
    pts, other = rng.uniform(0.0, 1.0, (n, ndim)), rng.uniform(0.0, 1.0, (700, ndim))
    k = Kernel("inv_r", 1.0 / n, 1.0)
    kw = dict(Nmax=nmax, eps_ACA=1e-8)
    M = HODLRdD_matrix(k, pts, *box, **kw).Assemble_matrix_operators()
    assert M.statistics()["n_far_blocks"] > 600000
    O = OracleHODLR(pts, *box, nmax=nmax, dprime=0, eps=1e-8, kind=1, scale=1.0 / n, diag=1.0, rng_mode=1)
    x = rng.uniform(0.5, 1.0, n)
    y, yo = M * x, O.matvec(x)
    assert np.array_equal(M.blocks()["rank"], O.blocks()["rank"])
    assert np.linalg.norm(y - yo) <= 1e-12 * np.linalg.norm(yo)
    assert np.array_equal(M * x, y)
    B = HODLRdD_batch([k, k], [pts, other], [box] * 2, **kw)
    X = torch.tensor(np.concatenate([x, rng.uniform(0.5, 1.0, 700)])[None], device="cuda")
    Y = torch.empty_like(X)
    B.matvec_device(X.data_ptr(), Y.data_ptr(), 1, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert np.array_equal(Y.cpu().numpy()[0, :n], y)
    S = HODLRdD_matrix(k, other, *box, **kw).Assemble_matrix_operators()
    assert np.array_equal(Y.cpu().numpy()[0, n:], S * X.cpu().numpy()[0, n:])
    for o in (M, B, S):
        o.close()
