"""Waits of the leaf-level tensor-core kernel that run out: a batch whose copies
never start (the message that is dropped), and a stage that one warp never hands
back.  Both are bounded by a few milliseconds here; the call reports
HODLR_ERR_DEVICE, and the next product on the same operator is the one from
before, bit for bit."""
import numpy as np
import pytest

from hodlrnd_gb300 import _lib
from hodlrnd_gb300.kernels import Kernel
from hodlrnd_gb300.matrix import HODLRdD_matrix

pytestmark = pytest.mark.gpu
WAIT_NS, DROP_COPIES, DROP_RELEASE = 0, 1, 2


@pytest.fixture(scope="module")
def operator():
    # 10 points a leaf and hundreds of sources a leaf, so that the leaf-level
    # kernel takes it, in runs of many batches
    n = 40000
    pts = np.random.default_rng(7).uniform(0.0, 1.0, (n, 4))
    M = HODLRdD_matrix(Kernel("inv_r2", 1.0 / n ** 0.5, 1.0), pts, [0.0] * 4, [1.0] * 4, Nmax=40, eps_ACA=1e-4,
                       precision="bf16_factors", fp64_check=False).Assemble_matrix_operators()
    yield M
    M.close()


@pytest.mark.parametrize("nrhs", [16, 32, 64])
@pytest.mark.parametrize("option,batch", [(DROP_COPIES, 0), (DROP_COPIES, 1), (DROP_COPIES, 2), (DROP_RELEASE, 0),
                                          (DROP_RELEASE, 1)])
def test_a_wait_that_runs_out_is_an_error(operator, option, batch, nrhs):
    torch = pytest.importorskip("torch")
    M = operator
    X = torch.randn((nrhs, M.N), dtype=torch.float32, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    Y, Z = torch.empty_like(X), torch.empty_like(X)
    M.matvec_tc_device(X.data_ptr(), Y.data_ptr(), nrhs)
    L = _lib.lib()
    for o, v in ((WAIT_NS, 5_000_000), (option, batch)):
        _lib.check(L.hodlr_test_option(M._op, o, v))
    with pytest.raises(_lib.HodlrError):
        M.matvec_tc_device(X.data_ptr(), Z.data_ptr(), nrhs)
    for o in (WAIT_NS, option):
        _lib.check(L.hodlr_test_option(M._op, o, -1))
    M.matvec_tc_device(X.data_ptr(), Z.data_ptr(), nrhs)
    assert torch.equal(Y, Z)
