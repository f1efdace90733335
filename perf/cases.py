"""The work that users of mpdok_gb300 have it do, as cases that can be timed and compared.

Every case goes through the package's public entry points.  Systems are the
ones of ``mpdok_gb300.configs``: Gaussian RBF interpolation on stratified or
uniform centres, nugget 1e-2, a white-noise right-hand side.  The shape
parameter follows the point density (gamma = 1600 at N = 32768, the headline
system), so a system of any size has about the headline's conditioning and
its solution is well determined.

Kinds of case:

* ``solve``     MixedSolver.solve: low-precision LU, FP32 GMRES, FP64 refinement
* ``lu_ir``     LUIRSolver.solve: the drop-in FP32 LU with partial pivoting
* ``multi_rhs`` LUFactorization + solve_ir_many: factor once, many fields
* ``gmres_ir``  MPDOKSolver.solve: the drop-in GMRES-IR
* ``matvec``    one FP32 product: DenseLinearOperator.matvec (stored) or MatrixFreeOperator.matvec
* ``assemble``  build_rbf_kernel: one kernel matrix
* ``evaluate``  rbf_evaluate: the interpolant at query points
* ``batch``     rbf_batch_solve, forward and backward: a training step
* ``grad``      rbf_solve, forward and backward: one differentiated solve

The out-of-core solver is not among them: its passes are bound by the host
link, which other jobs share.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from mpdok_gb300.adjoint import rbf_solve
from mpdok_gb300.batch import BatchedRBFSolver, rbf_batch_solve
from mpdok_gb300.dense_krylov import DenseLinearOperator
from mpdok_gb300.lu import LUFactorization
from mpdok_gb300.matfree import MatrixFreeOperator, rbf_evaluate
from mpdok_gb300.mpdok_ops import LUIRSolver, MPDOKSolver
from mpdok_gb300.rbf_kernel import build_rbf_kernel
from mpdok_gb300.solvers import MixedSolver

REG = 1e-2                       # the nugget of the headline system and of the reference's demos
GAMMA_PER_POINT = 1600 / 32768   # the headline's shape parameter, per centre of the unit square
DTYPES = {"f64": torch.float64, "f32": torch.float32}


def listed():
    return [
        # the smallest solve: a first try, a unit test, a system per request; latency and launches count
        dict(name="solve-600-fp16", kind="solve", n=600, factors="fp16"),
        # an ordinary solve of odd size with BF16 factors (range instead of digits)
        dict(name="solve-9973-bf16", kind="solve", n=9973, factors="bf16"),
        # the headline system, the largest in daily use
        dict(name="solve-32768-fp16", kind="solve", n=32768, factors="fp16"),
        # FP32 factors: what users take when the kernel matrix is too ill conditioned for 16-bit factors
        dict(name="solve-16384-fp32", kind="solve", n=16384, factors="fp32"),
        # the reference's LU solver by name, pivoted, one system
        dict(name="lu_ir-5000", kind="lu_ir", n=5000),
        # time series on fixed sensors: one factorization, three fields at 24 times
        dict(name="multi_rhs-8192x72", kind="multi_rhs", n=8192, rhs=72),
        # the reference's main solver by name
        dict(name="gmres_ir-8192", kind="gmres_ir", n=8192),
        # one product of a user's own Krylov loop; the shortest call
        dict(name="matvec-2000", kind="matvec", n=2000, rhs=1, operator="stored"),
        # the kernel matrix of the largest 3-D system, FP64: every stored solve starts with one
        dict(name="assemble-20000-3d", kind="assemble", n=20000, dim=3, kernel="gaussian", dtype="f64"),
        # the fitted surface on a 128 x 128 grid, three fields
        dict(name="evaluate-20000x16384", kind="evaluate", n=20000, m=16384, rhs=3, dim=2,
             kernel="gaussian"),
        # fitting shape parameters, nuggets and centres of many small systems: one training step
        dict(name="batch-32", kind="batch", systems=32, lo=300, hi=4000, rhs=8, dim=2),
        # one larger system differentiated in all of its inputs
        dict(name="grad-6000-fp16", kind="grad", n=6000, factors="fp16"),
    ]


def _size(rng, lo, hi):
    """Log-uniform; sizes are as ragged as they come, a quarter of them multiples of 64."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(64, n // 64 * 64) if rng.random() < 0.25 else n


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "lu_ir", "multi_rhs", "gmres_ir", "matvec", "assemble", "evaluate",
                       "batch", "batch", "grad"])
    if kind == "solve":
        factors = rng.choice(["fp16", "bf16", "fp32"])
        return dict(kind=kind, n=_size(rng, 300, 16384 if factors == "fp32" else 32768), factors=factors)
    if kind == "lu_ir":
        return dict(kind=kind, n=_size(rng, 300, 6000))
    if kind == "multi_rhs":
        return dict(kind=kind, n=_size(rng, 500, 8192), rhs=rng.randint(2, 72))
    if kind == "gmres_ir":
        return dict(kind=kind, n=_size(rng, 300, 12000))
    if kind == "matvec":
        return dict(kind=kind, n=_size(rng, 500, 32768), rhs=rng.randint(1, 8),
                    operator=rng.choice(["stored", "matrix_free"]))
    if kind == "assemble":
        return dict(kind=kind, n=_size(rng, 500, 20000), dim=rng.choice([2, 3]),
                    kernel=rng.choice(["gaussian", "mq"]), dtype=rng.choice(["f64", "f64", "f32"]))
    if kind == "evaluate":
        return dict(kind=kind, n=_size(rng, 500, 20000), m=_size(rng, 100, 16384), rhs=rng.randint(1, 3),
                    dim=rng.choice([2, 3]), kernel=rng.choice(["gaussian", "mq"]))
    if kind == "batch":
        lo = rng.randint(100, 600)
        return dict(kind=kind, systems=rng.randint(1, 32), lo=lo, hi=_size(rng, lo + 100, 4000),
                    rhs=rng.randint(1, 8), dim=rng.choice([2, 3]))
    return dict(kind=kind, n=_size(rng, 300, 6000), factors=rng.choice(["fp16", "bf16", "fp32"]))


# ------------------------------------------------------------------- inputs

def _jittered(n, rng):
    """n of the cells of a square grid over [0, 1]^2, one point in each (host FP64)."""
    g = math.isqrt(n * 101 // 100 - 1) + 1
    cells = np.sort(rng.choice(g * g, n, replace=False))
    return (np.stack([cells // g, cells % g], axis=1) + rng.uniform(size=(n, 2))) / g


def _on_gpu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda")


def _gamma(case):
    """GMRES without a preconditioner is used where the kernel is narrow."""
    per_point = 2.0 / 3.0 if case["kind"] == "gmres_ir" else GAMMA_PER_POINT
    return per_point * case["n"]


def _batch_sizes(case):
    rng = np.random.default_rng(3)
    return [int(v) for v in rng.integers(case["lo"], case["hi"] + 1, size=case["systems"])]


def _inputs(case, seed):
    """The user's data, on the GPU, from the seed alone."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind in ("solve", "lu_ir", "gmres_ir", "grad", "multi_rhs"):
        n = case["n"]
        X = _on_gpu(_jittered(n, rng))
        b = _on_gpu(rng.standard_normal((case["rhs"], n))).t() if kind == "multi_rhs" else \
            _on_gpu(rng.standard_normal(n))
        d = dict(coords=X, b=b)
        if kind == "grad":
            d["grad_x"] = _on_gpu(rng.standard_normal(n))
        return d
    if kind == "matvec":
        x = _on_gpu(rng.standard_normal((case["rhs"], case["n"])).astype(np.float32)).t()
        return dict(coords=_on_gpu(_jittered(case["n"], rng)), x=x[:, 0] if case["rhs"] == 1 else x)
    if kind == "assemble":
        return dict(coords=_on_gpu(rng.uniform(size=(case["n"], case["dim"]))))
    if kind == "evaluate":
        return dict(coords=_on_gpu(rng.uniform(size=(case["n"], case["dim"]))),
                    query=_on_gpu(rng.uniform(size=(case["m"], case["dim"]))),
                    alpha=_on_gpu(rng.standard_normal((case["rhs"], case["n"]))).t())
    total = sum(_batch_sizes(case))
    return dict(coords=_on_gpu(rng.uniform(size=(total, case["dim"]))),
                eps=_on_gpu(rng.uniform(2.0, 8.0, size=case["systems"])),
                reg=_on_gpu(np.full(case["systems"], REG)),
                b=_on_gpu(rng.standard_normal(total * case["rhs"])),
                grad_x=_on_gpu(rng.standard_normal(total * case["rhs"])))


def prepare(case, seed):
    s = dict(case=case, **_inputs(case, seed))
    kind = case["kind"]
    if kind in ("solve", "lu_ir", "gmres_ir", "multi_rhs") or case.get("operator") == "stored":
        s["A"], _ = build_rbf_kernel(s["coords"], gamma=_gamma(case), reg=REG)
    if kind == "solve":
        s["solver"] = MixedSolver(factor_dtype=case["factors"])
    elif kind == "lu_ir":
        s["solver"] = LUIRSolver()
    elif kind == "gmres_ir":
        s["solver"] = MPDOKSolver()
    elif kind == "matvec":
        s["op"] = DenseLinearOperator(s.pop("A"), verbose=False) if case["operator"] == "stored" else \
            MatrixFreeOperator(s["coords"], gamma=_gamma(case), reg=REG)
    elif kind == "batch":
        s["sizes"] = _batch_sizes(case)
        s["solver"] = BatchedRBFSolver(s["sizes"], dim=case["dim"], nrhs=case["rhs"], grid_mult=2)
        for k in ("coords", "eps", "reg", "b"):
            s[k].requires_grad_(True)
    elif kind == "grad":
        s["eps"] = torch.tensor(math.sqrt(_gamma(case)), dtype=torch.float64, requires_grad=True)
        s["reg"] = torch.tensor(REG, dtype=torch.float64, requires_grad=True)
        for k in ("coords", "b"):
            s[k].requires_grad_(True)
    return s


# --------------------------------------------------------------------- runs

def run(state):
    s, case = state, state["case"]
    kind = case["kind"]
    if kind == "solve":
        x, _ = s["solver"].solve(s["A"], s["b"], tol=1e-12)
        return x
    if kind == "lu_ir":
        return s["solver"].solve(s["A"], s["b"], tol=1e-12, maxiter_outer=5)
    if kind == "multi_rhs":
        lu = LUFactorization(s["A"], dtype="fp32")
        X, _ = lu.solve_ir_many(s["A"], s["b"], tol=1e-12, maxiter_outer=5)
        return X
    if kind == "gmres_ir":
        return s["solver"].solve(s["A"], s["b"], tol=1e-12, maxiter_outer=20)
    if kind == "matvec":
        return s["op"].matvec(s["x"])
    if kind == "assemble":
        A, _ = build_rbf_kernel(s["coords"], gamma=100.0, reg=REG, kernel=case["kernel"], dtype=DTYPES[case["dtype"]])
        return A
    if kind == "evaluate":
        return rbf_evaluate(s["alpha"], s["coords"], s["query"], gamma=100.0, kernel=case["kernel"])
    if kind == "batch":
        X = rbf_batch_solve(s["coords"], s["eps"], s["reg"], s["b"], s["solver"])
    else:
        X = rbf_solve(s["coords"], s["eps"], s["reg"], s["b"], factor_dtype=case["factors"])
    grads = torch.autograd.grad(X, [s["coords"], s["eps"], s["reg"], s["b"]], s["grad_x"])
    return [X.detach(), *grads]


# --------------------------------------------------------- what a pass needs

def work(case):
    """Bytes of inputs and outputs, and the operations of the direct method
    (for an iteration: of one product)."""
    kind = case["kind"]
    if kind == "batch":
        # the mean over the sizes' range of n^2 and n^3, per system
        lo, hi, s, k = case["lo"], case["hi"], case["systems"], case["rhs"]
        m1, m2, m3 = (sum(v ** p for v in range(lo, hi + 1)) / (hi - lo + 1) for p in (1, 2, 3))
        per_entry = 2 * (2 * case["dim"] + 2) + 4 * k
        return dict(bytes=8.0 * s * m1 * (3 * k + 2 * case["dim"]),
                    flops=s * (m3 / 3 + 2 * 3 * 4 * m2 * k + per_entry * m2))
    n = float(case["n"])
    if kind == "solve":
        return dict(bytes=8 * n * n + 16 * n, flops=2 / 3 * n ** 3 + 4 * n * n)
    if kind == "lu_ir":
        return dict(bytes=8 * n * n + 16 * n, flops=2 / 3 * n ** 3 + 4 * n * n)
    if kind == "multi_rhs":
        k = case["rhs"]
        return dict(bytes=8 * n * n + 16 * n * k, flops=2 / 3 * n ** 3 + 4 * n * n * k)
    if kind == "gmres_ir":
        return dict(bytes=8 * n * n + 16 * n, flops=2 * n * n)
    if kind == "matvec":
        k = case["rhs"]
        if case["operator"] == "stored":
            return dict(bytes=4 * n * n + 8 * n * k, flops=2 * n * n * k)
        return dict(bytes=n * (16 + 8 * k), flops=n * n * (8 + 2 * k))
    if kind == "assemble":
        size = 8 if case["dtype"] == "f64" else 4
        return dict(bytes=size * n * n + 8 * n * case["dim"], flops=n * n * (3 * case["dim"] + 2))
    if kind == "evaluate":
        m, k, d = float(case["m"]), case["rhs"], case["dim"]
        return dict(bytes=8 * (n * (d + k) + m * (d + k)), flops=m * n * (3 * d + 2 + 2 * k))
    return dict(bytes=8 * (2 * 2 * n + 5 * n), flops=2 / 3 * n ** 3 + 30 * n * n)


# ------------------------------------------------------------------ 64 bits

def _r2(a, b):
    d = torch.zeros((a.shape[0], b.shape[0]), dtype=torch.float64, device=a.device)
    for k in range(a.shape[1]):
        d.add_((a[:, k, None] - b[None, :, k]).square_())
    return d


def _phi(r2, gamma, kernel="gaussian"):
    return r2.mul_(-gamma).exp_() if kernel == "gaussian" else r2.mul_(gamma).add_(1.0).sqrt_()


def _system(X, gamma):
    A = _phi(_r2(X, X), gamma)
    A.diagonal().add_(REG)
    return A


def _spd_solve(A, B):
    """Cholesky and one refinement, FP64."""
    L = torch.linalg.cholesky(A)
    X = torch.cholesky_solve(B, L)
    return X + torch.cholesky_solve(B - A @ X, L)


def _solve_with_gradients(C, eps, reg, B, G):
    """(X, dL/dC, dL/deps, dL/dreg, dL/dB) of A(C, eps, reg) X = B for dL/dX = G, dense FP64."""
    r2 = _r2(C, C)
    phi = torch.exp(-eps * eps * r2)
    A = phi + reg * torch.eye(C.shape[0], dtype=torch.float64, device=C.device)
    L = torch.linalg.cholesky(A)
    both = torch.cat([B, G], dim=1)
    Y = torch.cholesky_solve(both, L)
    Y = Y + torch.cholesky_solve(both - A @ Y, L)
    X, lam = Y[:, :B.shape[1]], Y[:, B.shape[1]:]
    M = -(lam @ X.t())
    S = (M + M.t()) * phi
    ge = (M * phi * r2).sum() * (-2.0 * eps)
    gc = -2.0 * eps * eps * (S.sum(dim=1, keepdim=True) * C - S @ C)
    return X, gc, ge, M.diagonal().sum(), lam


def exact(case, seed):
    d = _inputs(case, seed)
    kind = case["kind"]
    if kind in ("solve", "lu_ir", "gmres_ir"):
        return _spd_solve(_system(d["coords"], _gamma(case)), d["b"].reshape(-1, 1)).reshape(-1)
    if kind == "multi_rhs":
        return _spd_solve(_system(d["coords"], _gamma(case)), d["b"])
    if kind == "matvec":
        return _system(d["coords"], _gamma(case)) @ d["x"].to(torch.float64)
    if kind == "assemble":
        A = _phi(_r2(d["coords"], d["coords"]), 100.0, case["kernel"])
        A.diagonal().add_(REG)
        return A
    if kind == "evaluate":
        out = [_phi(_r2(q, d["coords"]), 100.0, case["kernel"]) @ d["alpha"] for q in d["query"].split(4096)]
        return torch.cat(out)
    if kind == "grad":
        X, gc, ge, gr, lam = _solve_with_gradients(d["coords"], math.sqrt(_gamma(case)), REG,
                                                   d["b"].reshape(-1, 1), d["grad_x"].reshape(-1, 1))
        return [X.reshape(-1), gc, ge, gr, lam.reshape(-1)]
    sizes = _batch_sizes(case)
    k, o = case["rhs"], 0
    Xs, gcs, ges, grs, lams = [], [], [], [], []
    for i, n in enumerate(sizes):
        B = d["b"][o * k:(o + n) * k].reshape(k, n).t()
        G = d["grad_x"][o * k:(o + n) * k].reshape(k, n).t()
        X, gc, ge, gr, lam = _solve_with_gradients(d["coords"][o:o + n], float(d["eps"][i]), REG, B, G)
        Xs.append(X.t().reshape(-1))
        gcs.append(gc)
        ges.append(ge)
        grs.append(gr)
        lams.append(lam.t().reshape(-1))
        o += n
    return [torch.cat(Xs), torch.cat(gcs), torch.stack(ges), torch.stack(grs), torch.cat(lams)]
