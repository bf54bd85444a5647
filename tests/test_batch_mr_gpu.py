"""The multi-right-hand-side kernels of FP32-vector batches at the sizes where
their lane tiles and stages can go wrong: leaves of 1 to 32 rows (1, 2 or 4 row
groups), panels just above 32 rows and above a 128-row tile, V chunks and U tiles
whose width is no multiple of 32, segments longer than a stage, instances of one
leaf, right-hand-side counts on both sides of 32.  Reference: each operator's own
FP64 product; FP32 factors, vectors and sums of at most a few thousand terms of
one sign stay within 1e-5 (2^-24 times the square root of the term count, with a
factor of 50), as in test_batch_gpu.py."""
import numpy as np
import pytest

from hodlrnd_gb300.batch import HODLRdD_batch
from hodlrnd_gb300.kernels import Kernel
from hodlrnd_gb300.matrix import HODLRdD_matrix

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("ndim,nmax,sizes,nrhs", [(3, 8, (1, 7, 1501, 3000), 32), (3, 33, (900, 2111), 1),
                                                  (2, 3, (700, 40), 33), (2, 100, (2500, 1300, 99), 31),
                                                  (3, 300, (4000, 301), 40), (1, 17, (1000, 18), 64)])
def test_mixed_batch_products(ndim, nmax, sizes, nrhs):
    rng = np.random.default_rng(nmax + nrhs)
    box = ([0.0] * ndim, [1.0] * ndim)
    inst = [(rng.uniform(0.0, 1.0, (n, ndim)), Kernel("inv_r", 1.0 / max(n, 2), 1.0)) for n in sizes]
    B = HODLRdD_batch([k for _, k in inst], [p for p, _ in inst], [box] * len(inst), Nmax=nmax, eps_ACA=1e-6, tol=1e-6,
                      precision="mixed", fp64_check=False)
    off = B.offsets
    X = torch.rand((nrhs, int(off[-1])), dtype=torch.float32, device="cuda",
                   generator=torch.Generator("cuda").manual_seed(nrhs)) + 0.5
    Y = torch.full_like(X, float("nan"))
    stream = torch.cuda.current_stream().cuda_stream
    B.matvec_device(X.data_ptr(), Y.data_ptr(), nrhs, stream)
    torch.cuda.synchronize()
    x, y = X.cpu().numpy().astype(np.float64), Y.cpu().numpy().astype(np.float64)
    for i, (p, k) in enumerate(inst):
        M = HODLRdD_matrix(k, p, *box, Nmax=nmax, eps_ACA=1e-6).Assemble_matrix_operators()
        for c in {0, nrhs // 2, nrhs - 1}:
            ref = M * x[c, off[i]:off[i + 1]]
            assert np.linalg.norm(y[c, off[i]:off[i + 1]] - ref) <= 1e-5 * np.linalg.norm(ref)
        M.close()
    Z = torch.empty_like(X)
    B.matvec_device(X.data_ptr(), Z.data_ptr(), nrhs, stream)
    torch.cuda.synchronize()
    assert torch.equal(Y, Z)
    B.close()
