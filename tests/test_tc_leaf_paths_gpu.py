"""The leaf-level tensor-core kernel at the sizes where it can go wrong, taken by
every case here (its run count says so) whatever the plan's own rule would choose:
leaves of 1 to 32 points, sources longer than a batch (above 160 points), groups
of panels at several levels, every instance of its right-hand-side counts (up to 16,
32, 64).  And the rule: operators on both sides of it.  Reference: the same stored
operator applied one column at a time; the two differ by the operand splitting and
the FP32 sums, 5e-5 at most, as in test_tc_matvec_gpu.py."""
import ctypes

import numpy as np
import pytest

from hodlrnd_gb300 import _lib
from hodlrnd_gb300.kernels import Kernel
from hodlrnd_gb300.matrix import HODLRdD_matrix

pytestmark = pytest.mark.gpu
TC_LEAF, LEAF_RUNS = 4, 2


def runs(M):
    v = ctypes.c_int64()
    _lib.check(_lib.lib().hodlr_test_value(M._op, LEAF_RUNS, ctypes.byref(v)))
    return v.value


def cloud(kind, ndim, n, rng):
    p = rng.uniform(0.0, 1.0, (n, ndim))
    if kind == "clustered":  # most points in one corner: small panels at several levels, long sources
        p[:n - n // 12] *= 0.07
    return p


def check(M, torch, nrhs, ks):
    n = M.N
    X = torch.randn((nrhs, n), dtype=torch.float32, device="cuda", generator=torch.Generator("cuda").manual_seed(nrhs))
    Y = torch.full_like(X, float("nan"))
    M.matvec_tc_device(X.data_ptr(), Y.data_ptr(), nrhs)
    x, y = X.cpu().numpy().astype(np.float64), Y.cpu().numpy().astype(np.float64)
    for k in ks:
        ref = M * x[k]
        assert np.linalg.norm(y[k] - ref) <= 5e-5 * np.linalg.norm(ref)


@pytest.mark.parametrize("kind,ndim,n,nmax,dprime", [
    ("uniform", 4, 9000, 128, 0), ("uniform", 3, 4100, 8, 0), ("uniform", 3, 9000, 32, 1), ("uniform", 2, 3000, 20, 0),
    ("uniform", 1, 700, 3, 0), ("uniform", 5, 4000, 64, 0), ("clustered", 3, 6000, 200, 0),
    ("clustered", 2, 5000, 300, -1), ("clustered", 2, 4000, 24, 0)])
def test_every_case_takes_the_kernel(kind, ndim, n, nmax, dprime):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n + nmax)
    M = HODLRdD_matrix(Kernel("exp_neg_r", 1.0 / n ** 0.5, 1.0), cloud(kind, ndim, n, rng), [0.0] * ndim, [1.0] * ndim,
                       Nmax=nmax, eps_ACA=1e-4, INTERACTION_TYPE_ALLOWED=dprime, precision="bf16_factors",
                       fp64_check=False).Assemble_matrix_operators()
    _lib.check(_lib.lib().hodlr_test_option(M._op, TC_LEAF, 1))
    for nrhs in (1, 16, 17, 33, 48, 64):
        check(M, torch, nrhs, {0, nrhs - 1})
        assert runs(M) > 0
    t, b = M.tree_structure(), M.blocks()
    if kind == "clustered" and nmax >= 200:  # far sources longer than a batch in panels of at most 32 rows
        first = np.concatenate([[0], np.cumsum(t["level_sizes"])])
        m, s = t["node_counts"][first[b["level"]] + b["t"]], t["node_counts"][first[b["level"]] + b["s"]]
        assert ((m <= 32) & (s > 160) & (b["rank"] > 0)).any()
    M.close()


@pytest.mark.parametrize("ndim,n,nmax,dprime,taken", [
    (4, 5000, 40, -1, True), (4, 3000, 128, 0, True), (3, 9000, 64, 0, True), (3, 5000, 64, 0, True),
    (3, 3000, 64, 0, False), (3, 20000, 64, 0, False), (2, 5000, 64, 0, False), (4, 9000, 128, 0, False)])
def test_where_the_rule_lies(ndim, n, nmax, dprime, taken):
    torch = pytest.importorskip("torch")
    kind = {2: "log_r", 3: "inv_r", 4: "inv_r2"}[ndim]
    scale = {2: 1.0 / n, 3: n ** (-2.0 / 3.0), 4: n ** -0.5}[ndim]
    pts = np.random.default_rng(n).uniform(0.0, 1.0, (n, ndim))
    M = HODLRdD_matrix(Kernel(kind, scale, 1.0), pts, [0.0] * ndim, [1.0] * ndim, Nmax=nmax, eps_ACA=1e-4,
                       INTERACTION_TYPE_ALLOWED=dprime, precision="bf16_factors",
                       fp64_check=False).Assemble_matrix_operators()
    check(M, torch, 64, {0, 63})
    assert (runs(M) > 0) == taken
    M.close()
