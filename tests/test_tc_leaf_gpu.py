"""The leaf-level kernel of the tensor-core products (panels of at most 32 rows)
at the sizes where it can go wrong: leaves of 1 to 32 points on both sides of its
8-row and 8-point pieces, sources longer than a batch, panels with few
neighbours, groups that span levels (clustered points), right-hand-side counts
around its groups of 16.  Reference: the same stored operator applied one column
at a time; as in test_tc_matvec_gpu.py the two differ by the operand splitting
and the FP32 sums, 5e-5 at most."""
import numpy as np
import pytest

from hodlrnd_gb300.kernels import Kernel
from hodlrnd_gb300.matrix import HODLRdD_matrix

pytestmark = pytest.mark.gpu


def clouds(kind, ndim, n, rng):
    p = rng.uniform(0.0, 1.0, (n, ndim))
    if kind == "clustered":  # most points in one corner: small panels at several levels, long sources
        k = n - n // 12
        p[:k] *= 0.07
    return p


@pytest.mark.parametrize("kind,ndim,n,nmax,dprime,nrhs", [
    ("uniform", 4, 9000, 128, 0, 64), ("uniform", 4, 5000, 40, -1, 17), ("uniform", 3, 4100, 8, 0, 33),
    ("uniform", 3, 9000, 32, 1, 16), ("uniform", 2, 3000, 20, 0, 1), ("uniform", 1, 700, 3, 0, 5),
    ("clustered", 3, 6000, 200, 0, 48), ("clustered", 2, 5000, 300, -1, 64), ("uniform", 5, 4000, 64, 0, 32)])
def test_leaf_products(kind, ndim, n, nmax, dprime, nrhs):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n + nrhs)
    pts = clouds(kind, ndim, n, rng)
    M = HODLRdD_matrix(Kernel("exp_neg_r", 1.0 / n ** 0.5, 1.0), pts, [0.0] * ndim, [1.0] * ndim, Nmax=nmax, eps_ACA=1e-4,
                       INTERACTION_TYPE_ALLOWED=dprime, precision="bf16_factors",
                       fp64_check=False).Assemble_matrix_operators()
    X = torch.randn((nrhs, n), dtype=torch.float32, device="cuda", generator=torch.Generator("cuda").manual_seed(nrhs))
    Y = torch.full_like(X, float("nan"))
    M.matvec_tc_device(X.data_ptr(), Y.data_ptr(), nrhs)
    x, y = X.cpu().numpy().astype(np.float64), Y.cpu().numpy().astype(np.float64)
    for k in {0, nrhs // 2, nrhs - 1}:
        ref = M * x[k]
        assert np.linalg.norm(y[k] - ref) <= 5e-5 * np.linalg.norm(ref)
    Z = torch.empty_like(X)
    M.matvec_tc_device(X.data_ptr(), Z.data_ptr(), nrhs)
    assert torch.equal(Y, Z)
    M.close()
