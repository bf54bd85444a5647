"""The output rows of an FP32-vector batch are the FP64 sums of their slots (near
field and levels), also where a slot holds an infinity or the sum passes FP32's
range on the way: a row whose near field overflows is infinite and no NaN, and
the rows whose slots stay finite are those of the operator's own product."""
import numpy as np
import pytest

from hodlrnd_gb300.batch import HODLRdD_batch
from hodlrnd_gb300.kernels import Kernel
from hodlrnd_gb300.matrix import HODLRdD_matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrhs", [1, 5, 33])
def test_rows_beyond_fp32(nrhs):
    torch = pytest.importorskip("torch")
    n, box = 700, ([0.0] * 2, [1.0] * 2)
    pts = np.random.default_rng(3).uniform(0.0, 1.0, (n, 2))
    k = Kernel("inv_r", 1e-5, 2.0)  # diagonal 2: |2 x| passes 3.4e38 where |x| = 3e38
    B = HODLRdD_batch([k], [pts], [box], Nmax=32, eps_ACA=1e-6, tol=1e-6, precision="mixed", fp64_check=False)
    M = HODLRdD_matrix(k, pts, *box, Nmax=32, eps_ACA=1e-6).Assemble_matrix_operators()
    x = np.random.default_rng(4).uniform(-1.0, 1.0, (nrhs, n)).astype(np.float32)
    big = {7: 3e38, 300: -3e38, 699: 3e38}
    for i, v in big.items():
        x[:, i] = v
    X = torch.tensor(x, device="cuda")
    Y = torch.empty_like(X)
    B.matvec_device(X.data_ptr(), Y.data_ptr(), nrhs, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    y = Y.cpu().numpy()
    for c in {0, nrhs - 1}:
        assert np.array_equal(y[c, list(big)], np.sign(list(big.values())) * np.inf)
        ref = M * x[c].astype(np.float64)
        rest = np.abs(ref) < 3e38
        assert rest.sum() == n - len(big)
        assert np.linalg.norm(y[c, rest].astype(np.float64) / 1e30 - ref[rest] / 1e30) <= 1e-5 * np.linalg.norm(ref[rest] / 1e30)
    M.close()
    B.close()
