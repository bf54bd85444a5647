"""The largest blocks of a small build are compressed by clusters of CTAs, which
must return the factors of a single CTA to the last bit (norms are summed in
the same order): against hodlr_aca_block_noalloc, which takes a single CTA.
Sizes: node pieces of 32 points fewer than, equal to and more than the
cluster's warps, ragged; ranks beyond the first workspace (growth)."""
import ctypes

import numpy as np
import pytest

from hodlrnd_gb300 import _lib
from hodlrnd_gb300.kernels import Kernel
from hodlrnd_gb300.matrix import HODLRdD_matrix
from oracle.oracle import block_seed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ndim,n,eps", [(1, 1203, 1e-10), (2, 1100, 1e-12), (2, 8200, 1e-10), (3, 2405, 1e-8)])
def test_cluster_factors_are_those_of_a_cta(ndim, n, eps):
    torch = pytest.importorskip("torch")
    pts = np.random.default_rng(n).uniform(-1.0, 1.0, (n, ndim))
    M = HODLRdD_matrix(Kernel("inv_r", 1.0 / n, 1.0), pts, [-1.0] * ndim, [1.0] * ndim, Nmax=64,
                       eps_ACA=eps).Assemble_matrix_operators()
    B, S, perm = M.blocks(), M.tree_structure(), M.permutation()
    offs = np.concatenate([[0], np.cumsum(S["level_sizes"])])
    count = np.asarray(S["node_counts"])
    begin = np.concatenate([np.concatenate([[0], np.cumsum(count[a:b])[:-1]]) for a, b in zip(offs[:-1], offs[1:])])
    size = [max(count[offs[l] + t], count[offs[l] + s]) for l, t, s in zip(B["level"], B["t"], B["s"])]
    big = [b for b in np.argsort(size)[::-1][:3] if size[b] > 256]
    assert big
    P = ctypes.c_void_p
    fn = _lib.lib().hodlr_aca_block_noalloc
    fn.argtypes = [P, ctypes.c_int64, ctypes.c_int32, P, ctypes.c_int32, P, ctypes.c_int32,
                   ctypes.POINTER(_lib.HodlrKernelDesc), ctypes.c_double, ctypes.c_uint64, ctypes.c_int32, P,
                   ctypes.POINTER(ctypes.c_int32), ctypes.POINTER(ctypes.c_int32), P]
    fn.restype = ctypes.c_int
    d_points = torch.tensor(np.ascontiguousarray(pts.T), device="cuda")
    kd = _lib.HodlrKernelDesc(_lib.HODLR_KERNEL_INV_R, 0, 1.0 / n, 1.0)
    for b in big:
        l, t, s = int(B["level"][b]), int(B["t"][b]), int(B["s"][b])
        rows, cols = (perm[begin[offs[l] + k]:begin[offs[l] + k] + count[offs[l] + k]] for k in (t, s))
        m, k = len(rows), len(cols)
        cap = min(m, k, 512)
        d_rows, d_cols = (torch.tensor(np.sort(v).astype(np.int32), device="cuda") for v in (rows, cols))
        fac = torch.zeros((m + k) * cap, dtype=torch.float64, device="cuda")
        rank, flags = ctypes.c_int32(-1), ctypes.c_int32(-1)
        assert fn(d_points.data_ptr(), n, ndim, d_rows.data_ptr(), m, d_cols.data_ptr(), k, ctypes.byref(kd), eps,
                  block_seed(l, t, s), cap, fac.data_ptr(), ctypes.byref(rank), ctypes.byref(flags),
                  torch.cuda.current_stream().cuda_stream) == 0
        assert flags.value == 0 and rank.value == B["rank"][b]
        U, V, dense = M.block(b)
        assert not dense
        f, r = fac.cpu().numpy(), rank.value
        np.testing.assert_array_equal(U[np.argsort(rows, kind="stable")], f[:m * cap].reshape(cap, m).T[:, :r])
        np.testing.assert_array_equal(V[np.argsort(cols, kind="stable")], f[m * cap:].reshape(cap, k).T[:, :r])
    M.close()
