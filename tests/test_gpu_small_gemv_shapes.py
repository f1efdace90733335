"""GPU: the error-free FP64 product where the columns are split over blocks, and at the ends of its range."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _gemv(A, x, y, alpha, beta, lda=None):
    from mpdok_gb300 import _native as N
    from mpdok_gb300._device import ptr, stream_handle
    m, n = A.shape
    lib = N.load()
    size = lib.mpdok_gemv_workspace_size(N.F64, m, n, 1, 0)
    w = torch.full((size + 4096,), 0x5a, dtype=torch.uint8, device="cuda")
    N.check(lib.mpdok_gemv(N.F64, 0, ptr(A), lda or m, m, n, ptr(x), n, 1, ptr(y), m, alpha, beta, ptr(w), size,
                           stream_handle()), "gemv")
    assert torch.all(w[size:] == 0x5a)
    return y


@pytest.mark.parametrize("m,n", [(1, 255), (1, 256), (3, 257), (17, 4099), (8, 65536), (1, 524288), (300, 1500),
                                 (600, 600), (64, 1), (65, 1), (5792, 90), (8192, 64)])
def test_wide_and_tall_products(m, n):
    """y = -A x + b with b the rounded product.  With error-free sums one rounding of
    the result and n 2^-104 of |A| |x| (test_gpu_small_gemv.py); above 64 rows to a
    column the two-pass form, n 2^-53 of |A| |x|."""
    rng = np.random.default_rng(m + n)
    A, x = rng.standard_normal((m, n)), rng.standard_normal(n)
    b = A @ x
    y = _gemv(torch.from_numpy(np.asfortranarray(A)).cuda(), torch.from_numpy(x).cuda(), torch.from_numpy(b).cuda(), -1.0,
              1.0).cpu().numpy()
    c = 134217729.0
    xh = c * x - (c * x - x)
    xl = x - xh
    for i in sorted({0, m // 2, m - 1}):
        p = A[i] * x
        ah = c * A[i] - (c * A[i] - A[i])
        al = A[i] - ah
        e = ((ah * xh - p) + ah * xl + al * xh) + al * xl
        exact = math.fsum([b[i], *(-p), *(-e)])
        ax = float(np.abs(A[i]) @ np.abs(x))
        bound = 2.0 ** -52 * abs(exact) + (4 * n * 2.0 ** -105 if m <= 64 * n else n * 2.0 ** -53) * ax
        assert abs(y[i] - exact) <= bound


@pytest.mark.parametrize("m,n", [(16, 16), (8, 4096), (700, 700)])
def test_infinities_and_nan(m, n):
    A = torch.ones((n, m), dtype=torch.float64, device="cuda").t()
    A[m // 3, n - 1] = float("inf")
    A[m // 2, 0] = float("nan")
    A[m - 1, 0], A[m - 1, n - 1] = float("inf"), float("-inf")
    x = torch.ones(n, dtype=torch.float64, device="cuda")
    y = _gemv(A, x, torch.zeros(m, dtype=torch.float64, device="cuda"), 1.0, 0.0)
    ref = (A * x).sum(dim=1)
    assert torch.equal(torch.isnan(y), torch.isnan(ref))
    assert torch.equal(torch.nan_to_num(y, nan=0.0, posinf=1e300), torch.nan_to_num(ref, nan=0.0, posinf=1e300))


@pytest.mark.parametrize("n", [100, 600])
def test_residual_with_its_norm(n):
    """mpdok_residual: the norm of what it wrote, to the rounding of n additions, in one launch and in two."""
    from mpdok_gb300 import _native as N
    from mpdok_gb300._device import ptr, stream_handle
    rng = np.random.default_rng(n)
    A, b, x = (torch.from_numpy(rng.standard_normal(s)).cuda() for s in ((n, n), n, n))
    r, nrm = torch.empty_like(b), torch.zeros(1, dtype=torch.float64, device="cuda")
    lib = N.load()
    w = torch.empty(lib.mpdok_gemv_workspace_size(N.F64, n, n, 1, 0), dtype=torch.uint8, device="cuda")
    for _ in range(2):
        N.check(lib.mpdok_residual(ptr(A), n, n, ptr(b), ptr(x), ptr(r), ptr(nrm), ptr(w), w.numel(), stream_handle()), "residual")
    assert abs(nrm.item() - (r * r).sum().item()) <= 2 * n * 2.0 ** -53 * nrm.item()
    assert (r - (b - A.t() @ x)).abs().max().item() <= 4 * n * 2.0 ** -53 * (A.abs().t() @ x.abs()).max().item()


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("m,n,k", [(200000, 3, 1), (70000, 200, 3), (40000, 300, 8), (3000, 260, 1)])
def test_products_of_few_and_of_many_splits(m, n, k, dtype):
    """One to four splits (a thread adds an entry) and more: n u of |A| |X|, with
    rows that end inside a block."""
    from mpdok_gb300 import _native as N
    from mpdok_gb300._device import ptr, stream_handle
    g = torch.Generator("cuda").manual_seed(m)
    A = torch.randn(n, m, dtype=dtype, device="cuda", generator=g)
    X = torch.randn(k, n, dtype=dtype, device="cuda", generator=g)
    Y0 = torch.randn(k, m, dtype=dtype, device="cuda", generator=g)
    Y = Y0.clone()
    lib = N.load()
    code = N.F64 if dtype == torch.float64 else N.F32
    w = torch.empty(lib.mpdok_gemv_workspace_size(code, m, n, k, 0), dtype=torch.uint8, device="cuda")
    N.check(lib.mpdok_gemv(code, 0, ptr(A), m, m, n, ptr(X), n, k, ptr(Y), m, 1.5, -0.5, ptr(w), w.numel(),
                           stream_handle()), "gemv")
    ref = 1.5 * (X.double() @ A.double()) - 0.5 * Y0.double()
    bound = (n + 4) * torch.finfo(dtype).eps * (1.5 * (X.abs().double() @ A.abs().double()) + 0.5 * Y0.abs().double())
    assert torch.all((Y.double() - ref).abs() <= bound)


@pytest.mark.parametrize("n", [40, 300, 724])
@pytest.mark.parametrize("where", ["x", "column"])
def test_products_in_place(n, where):
    """y = x, or y a column of A: every entry is read before y is written (n u of |A| |x|)."""
    g = torch.Generator("cuda").manual_seed(n)
    S = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g)
    x = torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
    want, bound = S.t() @ x, n * 2.0 ** -52 * (S.abs().t() @ x.abs())
    for _ in range(3):
        A, v = S.clone().t(), x.clone()
        y = _gemv(A, v, v if where == "x" else A[:, n // 2], 1.0, 0.0)
        assert torch.all((y - want).abs() <= bound)
