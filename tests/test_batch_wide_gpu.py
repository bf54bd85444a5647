"""Blocks of an FP32-vector batch whose rank is above 128, the columns one item
takes, and above 1024: items of some of a row's columns, the last ones narrow.
Points in two neighbouring boxes of a 4D tree, so that the two blocks between
them have high ranks.  Reference: the operator's own FP64 product, to 1e-5 as in
test_batch_gpu.py."""
import numpy as np
import pytest

from hodlrnd_gb300.batch import HODLRdD_batch
from hodlrnd_gb300.kernels import Kernel
from hodlrnd_gb300.matrix import HODLRdD_matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,eps,ranks,nrhs", [(1200, 1e-4, (33, 300), 32), (2600, 1e-7, (129, 900), 7),
                                              (6000, 1e-12, (1024, 3000), 40)])
def test_wide_blocks(n, eps, ranks, nrhs):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    pts = rng.uniform(0.0, 1.0, (n, 4)) * np.array([1.0, 0.5, 0.5, 0.5])
    box = ([0.0] * 4, [1.0] * 4)
    k = Kernel("inv_r", 1.0 / n, 1.0)
    kw = dict(Nmax=n // 2 + n // 10, INTERACTION_TYPE_ALLOWED=3)
    B = HODLRdD_batch([k], [pts], [box], eps_ACA=eps, tol=1e-6, precision="mixed", fp64_check=False, **kw)
    M = HODLRdD_matrix(k, pts, *box, eps_ACA=eps, **kw).Assemble_matrix_operators()
    assert ranks[0] <= int(M.blocks()["rank"].max()) < ranks[1]
    X = torch.rand((nrhs, n), dtype=torch.float32, device="cuda", generator=torch.Generator("cuda").manual_seed(1)) + 0.5
    Y = torch.full_like(X, float("nan"))
    B.matvec_device(X.data_ptr(), Y.data_ptr(), nrhs, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    x, y = X.cpu().numpy().astype(np.float64), Y.cpu().numpy().astype(np.float64)
    for c in {0, nrhs - 1}:
        ref = M * x[c]
        assert np.linalg.norm(y[c] - ref) <= 1e-5 * np.linalg.norm(ref)
    M.close()
    B.close()
