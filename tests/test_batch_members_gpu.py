"""Each member of a batch is the operator built alone: its own products and
solves have the same bits, in every precision that batches take (the merged plan may cut the
members' work differently, their own plans may not)."""
import ctypes

import numpy as np
import pytest

from hodlrnd_gb300 import _lib
from hodlrnd_gb300.batch import HODLRdD_batch
from hodlrnd_gb300.kernels import Kernel
from hodlrnd_gb300.matrix import HODLRdD_matrix

pytestmark = pytest.mark.gpu
D = ctypes.POINTER(ctypes.c_double)


@pytest.mark.parametrize("precision", ["fp64", "fp32_factors", "mixed"])
def test_members_equal_operators_built_alone(precision):
    rng = np.random.default_rng(31)
    box = ([0.0] * 3, [1.0] * 3)
    inst = [(rng.uniform(0.0, 1.0, (n, 3)), Kernel("inv_r", 1.0 / n ** (2.0 / 3.0), 1.0)) for n in (300, 2111, 6000)]
    params = dict(Nmax=64, eps_ACA=1e-6, precision=precision, tol=1e-8)
    B = HODLRdD_batch([k for _, k in inst], [p for p, _ in inst], [box] * len(inst), **params)
    L = _lib.lib()
    for i, (p, k) in enumerate(inst):
        M = HODLRdD_matrix(k, p, *box, **params).Assemble_matrix_operators()
        b = rng.standard_normal(p.shape[0])
        y, x = np.empty_like(b), np.zeros_like(b)
        info = _lib.HodlrSolveInfo()
        _lib.check(L.hodlr_matvec(B.op(i), b.ctypes.data_as(D), y.ctypes.data_as(D), 1))
        assert np.array_equal(y, M * b)
        _lib.check(L.hodlr_solve(B.op(i), b.ctypes.data_as(D), x.ctypes.data_as(D), 1, ctypes.byref(info)))
        assert np.array_equal(x, M.solve(b))
        assert info.converged == 1 and info.iterations == M.last_solve["iterations"]
        M.close()
    B.close()
