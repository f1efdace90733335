"""GPU: the many-column residual where the digits of rows and columns would lose more than an FP64 product."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

N_, U = 2304, 2.0 ** -53


def _kernel(rng, n, gamma, reg):
    C = rng.uniform(0, 1, (n, 2))
    return np.exp(-gamma * ((C[:, None] - C[None]) ** 2).sum(-1)) + reg * np.eye(n)


def _split(a):
    t = a * 134217729.0
    h = t - (t - a)
    return h, a - h


def _true(A, X, B):
    """||B - A X|| per column, the products split into two doubles (Veltkamp, Dekker)
    and added pairwise with their rounding errors (some 2^-100 of the terms)."""
    out = []
    Ah, Al = _split(A)
    for c in range(B.shape[1]):
        x = X[:, c]
        xh, xl = _split(x)
        s = A * x
        e = ((Ah * xh - s) + Ah * xl + Al * xh) + Al * xl
        s, e = torch.cat([B[:, c:c + 1], -s], 1), torch.cat([torch.zeros_like(B[:, :1]), -e], 1)
        while s.shape[1] > 1:
            if s.shape[1] % 2:
                s, e = torch.nn.functional.pad(s, (0, 1)), torch.nn.functional.pad(e, (0, 1))
            p, q = s[:, 0::2], s[:, 1::2]
            t = p + q
            z = t - p
            e = (e[:, 0::2] + e[:, 1::2]) + ((p - (t - z)) + (q - z))
            s = t
        out.append((s + e).norm())
    return torch.stack(out)


@pytest.mark.parametrize("binades", [0, 15, 30])
@pytest.mark.parametrize("where", ["columns", "both", "one x"])
def test_reported_residual_stays_within_an_fp64_products_rounding(where, binades):
    """X = LU^-1 B without a refinement step, columns of A (or rows and columns,
    or one unknown) over +-binades: the reported ||B - A X|| / ||B|| is the true one
    to n u of || |A| |X| ||, the rounding of an FP64 product in any order."""
    from mpdok_gb300.lu import LUFactorization
    n, k = N_, 8
    rng = np.random.default_rng(binades)
    A = np.eye(n) + rng.standard_normal((n, n)) * (0.25 / np.sqrt(n))
    B = rng.standard_normal((n, k))
    if where == "one x":  # its column is small, so its x is large
        A[:, 7] *= 2.0 ** -binades
    else:
        A *= 2.0 ** rng.integers(-binades, binades + 1, n)
    if where == "both":
        A *= 2.0 ** rng.integers(-binades, binades + 1, n)[:, None]
    Ad, Bd = torch.from_numpy(np.asfortranarray(A)).cuda(), torch.from_numpy(np.asfortranarray(B)).cuda()
    lu = LUFactorization(Ad, dtype="fp32", pivoting=True)
    assert lu.info == 0
    X, info = lu.solve_ir_many(Ad, Bd, tol=1e-30, maxiter_outer=0)
    bn = Bd.norm(dim=0)
    true = _true(Ad, X, Bd) / bn
    off = n * U * (Ad.abs() @ X.abs()).norm(dim=0) / bn
    assert (true - off).max() <= info["history"][0][0][1] <= (true + off).max()


@pytest.mark.parametrize("decades", [0, 4, 6, 8])
@pytest.mark.parametrize("form,k,pivoting", [("KD", 8, True), ("DKD", 8, False), ("DKD", 20, True),
                                             ("DKD g", 8, True), ("DKD g", 20, False)])
def test_refinement_ends_where_the_fp64_product_lets_it(form, decades, k, pivoting):
    """K a Gaussian kernel matrix, D over some decades, right-hand sides g or D g:
    the residuals after six steps, to twice FP64, against the same columns
    solved three at a time (whose residual is the FP64 product).  Both end at the
    rounding of their residuals; three times the other's covers two roundings of
    equal size in either norm, with the spread of a worst column."""
    from mpdok_gb300 import _native as N
    from mpdok_gb300._device import fortran_empty, ptr, stream_handle
    from mpdok_gb300.lu import LUFactorization
    n = N_
    rng = np.random.default_rng(decades + k)
    K = _kernel(rng, n, 0.0488 * n, 1e-2)
    d = 10.0 ** rng.uniform(-decades / 2, decades / 2, n)
    A = K * d if form == "KD" else d[:, None] * K * d
    B = rng.standard_normal((n, k))
    if form == "DKD":
        B *= d[:, None]
    Ad, Bd = torch.from_numpy(np.asfortranarray(A)).cuda(), torch.from_numpy(np.asfortranarray(B)).cuda()
    lu = LUFactorization(Ad, dtype="fp32", pivoting=pivoting)
    X, info = lu.solve_ir_many(Ad, Bd, tol=1e-30, maxiter_outer=6)
    lib = N.load()
    Y = fortran_empty(n, k, torch.float64)
    for c in range(0, k, 3):
        kk = min(3, k - c)
        w = torch.empty(lib.mpdok_lu_ir_multi_work_size(n, kk), dtype=torch.uint8, device="cuda")
        one = N.SolveInfo()
        st = lib.mpdok_lu_ir_solve_multi(ptr(Ad), n, n, ptr(lu.factors), lu.fdtype, kk, ptr(Bd[:, c:c + kk]), n,
                                         ptr(Y[:, c:c + kk]), n, 1e-30, 6, ptr(w), w.numel(), ctypes.byref(one),
                                         stream_handle())
        assert st == 0, N.last_error()
    bn = Bd.norm(dim=0)
    many, few = _true(Ad, X, Bd) / bn, _true(Ad, Y, Bd) / bn
    assert many.max() <= 3 * few.max(), (many.max(), few.max())
    # the report tells the same (n u of the products, as above)
    off = n * U * (Ad.abs() @ X.abs()).norm(dim=0) / bn
    assert info["relres"] <= (many + off).max()


def test_zero_column_among_others():
    """A right-hand side of zeros drops nothing and keeps its group on the digits."""
    from mpdok_gb300.lu import LUFactorization
    n, k = 2048, 8
    rng = np.random.default_rng(1)
    A = _kernel(rng, n, 100.0, 0.1)
    B = rng.standard_normal((n, k))
    B[:, 3] = 0.0
    Ad, Bd = torch.from_numpy(A).cuda(), torch.from_numpy(np.asfortranarray(B)).cuda()
    X, info = LUFactorization(Ad, dtype="fp32").solve_ir_many(Ad, Bd, tol=1e-12, maxiter_outer=5)
    assert info["converged"] and torch.all(X[:, 3] == 0)
