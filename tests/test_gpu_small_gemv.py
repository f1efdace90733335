"""GPU: the one-launch FP64 product of small matrices is the rounded exact product."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,pad", [(1, 1, 0), (7, 31, 1), (8, 32, 0), (9, 33, 3), (130, 4, 0), (1, 5000, 2),
                                     (724, 724, 0), (5000, 104, 1)])
def test_small_fp64_gemv_is_the_rounded_exact_product(m, n, pad):
    """y = -A x + b with b the rounded product, so nearly everything cancels.
    The sums carry their rounding errors: one rounding of the result (2^-53)
    plus what the second-order terms leave, about n 2^-106 of |A| |x|."""
    from mpdok_gb300 import _native as N
    from mpdok_gb300._device import fortran_empty, ptr, stream_handle
    rng = np.random.default_rng(m + n)
    A = rng.standard_normal((m, n))
    x = rng.standard_normal(n)
    b = A @ x
    Ad = fortran_empty(m + pad, n, torch.float64)
    Ad[:m] = torch.from_numpy(A).cuda()
    xd, y = torch.from_numpy(x).cuda(), torch.from_numpy(b).cuda()
    lib = N.load()
    w = torch.empty(lib.mpdok_gemv_workspace_size(N.F64, m, n, 1, 0), dtype=torch.uint8, device="cuda")
    N.check(lib.mpdok_gemv(N.F64, 0, ptr(Ad), m + pad, m, n, ptr(xd), n, 1, ptr(y), m, -1.0, 1.0, ptr(w), w.numel(),
                           stream_handle()), "gemv")
    y = y.cpu().numpy()
    for i in range(m):
        # exact: every product split into two doubles (Veltkamp / Dekker), then fsum
        p = A[i] * x
        c = 134217729.0
        ah = c * A[i] - (c * A[i] - A[i])
        xh = c * x - (c * x - x)
        al, xl = A[i] - ah, x - xh
        e = ((ah * xh - p) + ah * xl + al * xh) + al * xl
        exact = math.fsum([b[i], *(-p), *(-e)])
        bound = 2.0 ** -52 * abs(exact) + 4 * n * 2.0 ** -105 * float(np.abs(A[i]) @ np.abs(x))
        assert abs(y[i] - exact) <= bound


def test_small_fp64_gemv_keeps_infinities():
    from mpdok_gb300 import _native as N
    from mpdok_gb300._device import ptr, stream_handle
    A = torch.ones((16, 16), dtype=torch.float64, device="cuda")
    A[3, 2] = float("inf")  # symmetric in layout: column-major reads entry (2, 3)
    A[5, 6] = float("nan")
    x = torch.ones(16, dtype=torch.float64, device="cuda")
    y = torch.empty_like(x)
    lib = N.load()
    w = torch.empty(lib.mpdok_gemv_workspace_size(N.F64, 16, 16, 1, 0), dtype=torch.uint8, device="cuda")
    N.check(lib.mpdok_gemv(N.F64, 0, ptr(A), 16, 16, 16, ptr(x), 16, 1, ptr(y), 16, 1.0, 0.0, ptr(w), w.numel(),
                           stream_handle()), "gemv")
    ref = A.cpu().t() @ torch.ones(16, dtype=torch.float64)
    assert torch.equal(torch.isnan(y.cpu()), torch.isnan(ref))
    assert torch.equal(torch.nan_to_num(y.cpu(), nan=0.0), torch.nan_to_num(ref, nan=0.0))
