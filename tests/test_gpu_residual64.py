"""GPU: the many-column FP64 residual on the tensor cores against extended precision."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,graded", [(2048, 4, False), (2111, 5, True), (2305, 8, True), (2050, 40, False)])
def test_reported_residual_is_the_true_one(n, k, graded):
    """X = LU^-1 B without a refinement step; the report's first entry is the worst
    ||B - A X|| / ||B|| of a group of eight.  Digit pairs below weight 7 are
    dropped: at most n 2^-57 of (largest of the row) x (largest of the column)
    per entry; the result is rounded once.  `graded`: rows and right-hand sides
    over 30 binades."""
    from mpdok_gb300.lu import LUFactorization
    rng = np.random.default_rng(n)
    A = np.eye(n) + rng.standard_normal((n, n)) * (0.25 / np.sqrt(n))
    B = rng.standard_normal((n, k))
    if graded:
        A *= 2.0 ** rng.integers(-15, 16, n)[:, None]
        B *= 2.0 ** rng.integers(-15, 16, k)
    Ad, Bd = torch.from_numpy(np.asfortranarray(A)).cuda(), torch.from_numpy(np.asfortranarray(B)).cuda()
    lu = LUFactorization(Ad, dtype="fp32", pivoting=True)
    X, info = lu.solve_ir_many(Ad, Bd, tol=1e-30, maxiter_outer=0)
    X = X.cpu().numpy()
    rowmax = np.abs(A).max(axis=1)
    Al = A.astype(np.longdouble)
    for q in sorted({0, (k - 1) // 8}):
        c = slice(8 * q, min(k, 8 * q + 8))
        R = B[:, c] - Al @ X[:, c].astype(np.longdouble)
        bn = np.linalg.norm(B[:, c], axis=0)
        true = np.linalg.norm(R.astype(np.float64), axis=0) / bn
        off = n * 2.0 ** -57 * np.linalg.norm(rowmax) * np.abs(X[:, c]).max(axis=0) / bn + 2.0 ** -50 * true
        reported = info["history"][q][0][1]
        assert np.max(true - off) <= reported <= np.max(true + off)


def test_refinement_reaches_below_the_fp64_products_rounding():
    """With exact products the refinement ends at the rounding of X itself."""
    from mpdok_gb300.lu import LUFactorization
    rng = np.random.default_rng(5)
    n, k = 2200, 16
    C = rng.uniform(0, 1, (n, 2))
    A = np.exp(-200.0 * ((C[:, None] - C[None]) ** 2).sum(-1)) + 1e-2 * np.eye(n)
    B = rng.standard_normal((n, k))
    Ad, Bd = torch.from_numpy(A).cuda(), torch.from_numpy(np.asfortranarray(B)).cuda()
    lu = LUFactorization(Ad, dtype="fp32")
    X, info = lu.solve_ir_many(Ad, Bd, tol=1e-30, maxiter_outer=8)
    # the rounded solution's own residual: half an ulp of every entry, random signs
    bound = 2 * 2.0 ** -53 * (torch.linalg.matrix_norm(Ad, 2) * X.norm(dim=0) / Bd.norm(dim=0)).max().item()
    assert info["relres"] <= bound


def test_non_finite_matrix_is_reported():
    from mpdok_gb300 import _native as N
    from mpdok_gb300.lu import LUFactorization
    rng = np.random.default_rng(6)
    n = 2048
    A = np.eye(n) + rng.standard_normal((n, n)) * (0.25 / np.sqrt(n))
    Ad, Bd = torch.from_numpy(A).cuda().t(), torch.from_numpy(np.asfortranarray(rng.standard_normal((n, 8)))).cuda()
    lu = LUFactorization(Ad, dtype="fp32")
    Ad[5, 7] = float("inf")
    with pytest.raises(N.MPDOKError) as e:
        lu.solve_ir_many(Ad, Bd, tol=1e-12)
    assert e.value.status == N.ERR_NONFINITE
