"""The work that a program using this engine has it do, case by case: the
operator's product with one vector, with a block of vectors on the tensor
cores and for a batch of operators, the GMRES solve, and the build.

Operators are described by their dimension, size, kernel, admissibility
(dprime), leaf size, tolerance and precision; points are uniform in a box and
vectors N(0, 1), as in the benchmark's workloads.
"""
import ctypes
import math

import numpy as np
import torch

from hodlrnd_gb300 import Kernel, _lib
from hodlrnd_gb300.batch import HODLRdD_batch
from hodlrnd_gb300.matrix import HODLRdD_matrix


def _case(do, ndim, n, precision, eps, **more):
    c = dict(do=do, ndim=ndim, n=n, precision=precision, eps=eps, kind="inv_r", nmax=64, dprime=0, nrhs=1, host=False,
             check=False, tol=eps, seed_shift=0)
    c.update(more)
    return c


def listed():
    out = []

    def add(name, *a, **k):
        out.append(dict(_case(*a, **k), name=name))

    # A small operator applied through host arrays (`M * x`): what a script or a
    # test does, where copies, launches and host work are all there is.
    add("product_2d_n2000_fp64_host", "product", 2, 2000, "fp64", 1e-10, host=True)
    # The 2D configuration, FP64, vectors on the device: one step of a caller's own iteration.
    add("product_2d_n10000_fp64", "product", 2, 10000, "fp64", 1e-10)
    # A middling 3D operator of a size that is no power of two, in the reference's own arithmetic.
    add("product_3d_n30011_fp64", "product", 3, 30011, "fp64", 1e-8)
    # The 3D configuration at full size, FP32-stored factors, products at FP64 level.
    add("product_3d_n262144_fp32", "product", 3, 262144, "fp32_factors", 1e-8)
    # The 4D configuration: BF16 column-scaled factors at a loose tolerance, larger leaves.
    add("product_4d_n65536_bf16", "product", 4, 65536, "bf16_factors", 1e-4, kind="inv_r2", nmax=128)
    # The same operator applied to 64 vectors at once (tensor cores).
    add("block_4d_n65536_bf16_64rhs", "block", 4, 65536, "bf16_factors", 1e-4, kind="inv_r2", nmax=128, nrhs=64)
    # Independent 3D operators, log-uniform sizes, 32 FP32 vectors each: the batched workload, fewer instances.
    add("batch_3d_24x_mixed_32rhs", "batch", 3, 24, "mixed", 1e-6, nrhs=32)
    # The 2D configuration solved in FP64 from host arrays, as the reference's main program does.
    add("solve_2d_n10000_fp64_host", "solve", 2, 10000, "fp64", 1e-10, host=True)
    # A request of the serving workload: a middling 3D geometry that is resident, a few right-hand
    # sides from host arrays.  Solves are taken to 1e-11, below the compression error.
    add("solve_3d_n20011_fp32_3rhs_host", "solve", 3, 20011, "fp32_factors", 1e-8, nrhs=3, host=True, check=True, tol=1e-11)
    # The 3D configuration at full size: one solve on the resident operator.
    add("solve_3d_n262144_fp32", "solve", 3, 262144, "fp32_factors", 1e-8, check=True, tol=1e-11)
    # Builds: a new geometry arrives.  Small (launches, host passes) and large (compression itself).
    add("build_2d_n10000_fp64", "build", 2, 10000, "fp64", 1e-10, host=True)
    add("build_3d_n100003_fp32", "build", 3, 100003, "fp32_factors", 1e-8, check=True, host=True)
    return out


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    do = rng.choice(["product"] * 4 + ["block", "batch", "solve", "solve", "build", "build"])
    shift = rng.randrange(1 << 20)
    if do == "batch":
        return _case(do, 3, rng.randrange(2, 25), "mixed", 1e-6, nrhs=rng.randrange(1, 41), seed_shift=shift)
    if do == "block":
        ndim = rng.choice([2, 3, 4])
        return _case(do, ndim, _log_size(rng, 3000, 65536), "bf16_factors", 1e-4,
                     kind={2: "log_r", 3: "inv_r", 4: "inv_r2"}[ndim], nmax=128 if ndim == 4 else 64,
                     dprime=rng.choice([-1, 0]), nrhs=rng.randrange(1, 97), seed_shift=shift)
    precision = rng.choice(["fp64", "fp32_factors", "fp32_factors", "bf16_factors", "mixed"])
    if do == "solve":
        # kernels and scalings of the 2D and 3D configurations: GMRES converges on them at every size
        ndim = rng.choice([2, 3])
        host = rng.random() < 0.5
        return _case(do, ndim, _log_size(rng, 1500, 65536), precision, 1e-8, check=True, tol=1e-11, host=host,
                     nrhs=rng.choice([1, 1, 2, 3]), seed_shift=shift)
    ndim = rng.choice([2, 3, 3, 4])
    kind = rng.choice(["inv_r", "exp_neg_r"] + (["log_r"] if ndim == 2 else []) + (["inv_r2"] if ndim == 4 else []))
    eps = 1e-4 if precision == "bf16_factors" else rng.choice([1e-6, 1e-8, 1e-10])
    if do == "build":
        n = _log_size(rng, 1500, {2: 65536, 3: 50000, 4: 16384}[ndim])
    else:
        n = _log_size(rng, 1500, {2: 262144, 3: 200000, 4: 32768}[ndim])
    return _case(do, ndim, n, precision, eps, kind=kind, nmax=128 if ndim == 4 else rng.choice([32, 64, 64, 100]),
                 dprime=rng.choice([-1, 0, 0]), check=do == "build" and precision != "fp64" and rng.random() < 0.5,
                 host=do == "build" or rng.random() < 0.3, nrhs=1, seed_shift=shift)


# ---------------------------------------------------------------- inputs
def _box(ndim):
    return ([-1.0] * 2, [1.0] * 2) if ndim == 2 else ([0.0] * ndim, [1.0] * ndim)


def _points(ndim, n, rng):
    lo, hi = _box(ndim)
    return rng.uniform(lo[0], hi[0], (n, ndim))


def _scale(ndim, n, kind):
    # 1/N in 2D and N^-((d-1)/d) in 3D; in 4D N^-1/2 for 1/r^2
    if ndim == 2:
        return 1.0 / n
    if ndim == 4 and kind == "inv_r2":
        return 1.0 / n ** 0.5
    return 1.0 / n ** ((ndim - 1) / ndim)


def _instances(case, seed):
    """[(points, scale)]: one for a single operator, several for a batch."""
    rng = np.random.default_rng([seed, case["seed_shift"]])
    if case["do"] != "batch":
        n = case["n"]
        return [(_points(case["ndim"], n, rng), _scale(case["ndim"], n, case["kind"]))]
    ns = [int(round(math.exp(v))) for v in
          np.random.default_rng([case["n"], case["seed_shift"]]).uniform(math.log(2048), math.log(65536), case["n"])]
    return [(_points(case["ndim"], n, rng), _scale(case["ndim"], n, case["kind"])) for n in ns]


def _params(case):
    return dict(Nmax=case["nmax"], eps_ACA=case["eps"], INTERACTION_TYPE_ALLOWED=case["dprime"],
                precision=case["precision"], tol=case["tol"], fp64_check=case["check"])


def _vectors(case, seed, n):
    """(nrhs, n): each row one column of the n x nrhs column-major block."""
    single = case["do"] in ("batch", "block")
    g = torch.Generator(device="cuda").manual_seed(seed * 7919 + 17)
    return torch.randn((case["nrhs"], n), dtype=torch.float32 if single else torch.float64, device="cuda", generator=g)


def _matrix(case, seed):
    pts, scale = _instances(case, seed)[0]
    return HODLRdD_matrix(Kernel(case["kind"], scale, 1.0), pts, *_box(case["ndim"]), **_params(case))


def prepare(case, seed):
    s = dict(case=case)
    if case["do"] == "batch":
        inst = _instances(case, seed)
        s["op"] = HODLRdD_batch([Kernel(case["kind"], sc, 1.0) for _, sc in inst], [p for p, _ in inst],
                                [_box(case["ndim"])] * len(inst), **_params(case))
        n = int(s["op"].offsets[-1])
    else:
        s["op"] = _matrix(case, seed)
        if case["do"] != "build":
            s["op"].Assemble_matrix_operators()
        n = case["n"]
    x = _vectors(case, seed, n)
    if case["host"]:
        x = x.cpu().numpy()
        s["x"] = x[0].copy() if case["nrhs"] == 1 else x.T  # (n,) or Fortran-ordered (n, nrhs)
    else:
        s["x"], s["y"] = x, torch.empty_like(x)
    return s


def run(s):
    case, op, x = s["case"], s["op"], s["x"]
    do = case["do"]
    if do == "build":
        op.Assemble_matrix_operators()
        return {"y": op * x, "order": op.permutation()}
    if case["host"]:
        return op.solve(x) if do == "solve" else op * x
    y, nrhs = s["y"], case["nrhs"]
    stream = torch.cuda.current_stream().cuda_stream
    if do == "solve":
        op.solve_device(x.data_ptr(), y.data_ptr(), nrhs, stream)
    elif do == "block":
        op.matvec_tc_device(x.data_ptr(), y.data_ptr(), nrhs, stream)
    else:
        op.matvec_device(x.data_ptr(), y.data_ptr(), nrhs, stream)
    return y


# ---------------------------------------------------------------- what a pass cannot do without
def _stored(case, stats):
    """(bytes, entries) of one operator's factors, each entry once."""
    far = {"fp64": 8, "fp32_factors": 4, "mixed": 4, "bf16_factors": 2}[case["precision"]]
    near = 4 if case["do"] == "batch" else 8
    entries = stats["far_entries"] + stats["dense_far_entries"]
    return entries * far + stats["near_entries"] * near, entries + stats["near_entries"]


def _aca_flops(op, ndim):
    """Entries, residual subtractions and norm estimates of the compression."""
    t, b = op.tree_structure(), op.blocks()
    first = np.concatenate([[0], np.cumsum(t["level_sizes"])])
    counts = t["node_counts"]
    mn = (counts[first[b["level"]] + b["t"]] + counts[first[b["level"]] + b["s"]]).astype(np.float64)
    r = b["rank"].astype(np.float64)
    return float(np.sum(mn * ((r + 1) * (3 * ndim + 2) + 2 * r * r)))


def work(case):
    nrhs = case["nrhs"]
    if case["do"] == "batch":
        s = prepare(case, 1)
        stored = entries = 0.0
        for i in range(s["op"].count):
            st = _lib.HodlrStats()
            _lib.check(_lib.lib().hodlr_stats_get(s["op"].op(i), ctypes.byref(st)))
            b, e = _stored(case, st.as_dict())
            stored, entries = stored + b, entries + e
        n = int(s["op"].offsets[-1])
        s["op"].close()
        return {"bytes": stored + 2 * 4 * n * nrhs, "flops": 2 * entries * nrhs}
    M, n = _matrix(case, 1), case["n"]
    M.Assemble_matrix_operators()
    stored, entries = _stored(case, M.statistics())
    if case["do"] == "build":
        copies = stored + (8 * (M.statistics()["far_entries"] + M.statistics()["dense_far_entries"]) if case["check"] else 0)
        w = {"bytes": copies + 8 * n * (case["ndim"] + 2) + stored, "flops": _aca_flops(M, case["ndim"]) + 2 * entries}
    elif case["do"] == "solve":
        # a product and the orthogonalisation against the basis so far, each iteration
        M.solve(_vectors(case, 1, n).cpu().numpy().T)
        its = max(1, M.last_solve["iterations"])
        its = its if nrhs == 1 else its / nrhs
        basis = 8 * n * min(its, 100) / 2 * 2
        w = {"bytes": nrhs * its * (stored + basis), "flops": nrhs * its * (2 * entries + 4 * n * min(its, 100) / 2)}
    else:
        vec = 4 if case["do"] == "block" else 8
        w = {"bytes": stored + 2 * vec * n * nrhs, "flops": 2 * entries * nrhs}
    M.close()
    return w


# ---------------------------------------------------------------- in 64 bits
def _dense_rows(P, i0, i1, kind, scale):
    d2 = torch.zeros((i1 - i0, P.shape[0]), dtype=torch.float64, device=P.device)
    for k in range(P.shape[1]):
        t = P[i0:i1, k, None] - P[None, :, k]
        d2.addcmul_(t, t)
        del t
    i = torch.arange(i0, i1, device=P.device)
    d2[i - i0, i] = 1.0
    if kind == "inv_r":
        a = d2.sqrt_().reciprocal_().mul_(scale)
    elif kind == "inv_r2":
        a = d2.reciprocal_().mul_(scale)
    elif kind == "log_r":
        a = d2.sqrt_().log_().mul_(scale)
    else:
        a = d2.sqrt_().neg_().exp_().mul_(scale)
    a[i - i0, i] = 1.0
    return a


def _dense_product(pts, kind, scale, X):
    """(nrhs, n) = X A^T for the dense kernel matrix, rows in chunks."""
    P = torch.tensor(pts, device="cuda")
    n = P.shape[0]
    Y = torch.empty(X.shape, dtype=torch.float64, device="cuda")
    step = max(1, (1 << 28) // n)
    for i0 in range(0, n, step):
        i1 = min(n, i0 + step)
        Y[:, i0:i1] = X @ _dense_rows(P, i0, i1, kind, scale).T
    return Y


def exact(case, seed):
    inst = _instances(case, seed)
    n = sum(p.shape[0] for p, _ in inst)
    X = _vectors(case, seed, n).double()
    if case["do"] == "solve":
        if n > 16000:
            return None
        P = torch.tensor(inst[0][0], device="cuda")
        A = _dense_rows(P, 0, n, case["kind"], inst[0][1])
        Y = torch.linalg.solve(A, X.T).T
    else:
        Y, at = torch.empty_like(X), 0
        for p, scale in inst:
            Y[:, at:at + p.shape[0]] = _dense_product(p, case["kind"], scale, X[:, at:at + p.shape[0]].contiguous())
            at += p.shape[0]
    if case["host"]:
        Y = Y.cpu().numpy()
        Y = Y[0] if case["nrhs"] == 1 else Y.T
    return {"y": Y, "order": None} if case["do"] == "build" else Y
