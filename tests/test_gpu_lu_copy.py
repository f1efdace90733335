"""The factorization that also writes A rounded to FP32: the copy's bits, and the same factors."""
import pytest
import torch

from mpdok_gb300 import _native as N

pytestmark = pytest.mark.gpu


def _factor(A, n, lda, fdtype, pivoting, ld32):
    from mpdok_gb300._device import ptr, stream_handle
    lib = N.load()
    f = torch.zeros(lib.mpdok_lu_factor_size(n, fdtype), dtype=torch.uint8, device="cuda")
    w = torch.empty(lib.mpdok_lu_work_size(n, fdtype), dtype=torch.uint8, device="cuda")
    A32 = torch.full((n, max(1, ld32)), 7.0, device="cuda") if ld32 else None
    N.check(lib.mpdok_lu_factor_copy(ptr(A), lda, n, fdtype, pivoting, ptr(f), f.numel(), ptr(w), w.numel(), ptr(A32),
                                     ld32, stream_handle()))
    return f, A32


@pytest.mark.parametrize("pivoting", [0, 1])
@pytest.mark.parametrize("n", [1, 4, 5, 130, 1028, 2047, 2052])
def test_copy_and_factors(n, pivoting):
    g = torch.Generator().manual_seed(n)
    M = torch.randn(n, n, generator=g, dtype=torch.float64) / n
    M.diagonal().add_(2.0 + torch.rand(n, generator=g, dtype=torch.float64))
    even, base = (n + 3) // 4 * 4, None
    # (lda, lda32): whole vectors; an odd lda; an odd lda32; no copy
    for lda, ld32 in ((even, even), (even + 1, even), (even, even + 1), (even, 0)):
        A = torch.zeros(n, lda, dtype=torch.float64)
        A[:, :n] = M
        f, A32 = _factor(A.cuda(), n, lda, N.F16, pivoting, ld32)
        base = f if base is None else base
        assert torch.equal(f, base)
        if ld32:
            A32 = A32.cpu()
            assert torch.equal(A32[:, :n], M.float())
            assert (A32[:, n:] == 7.0).all()


def test_copy_pitch_is_checked():
    from mpdok_gb300._device import ptr, stream_handle
    lib = N.load()
    A = torch.eye(8, dtype=torch.float64, device="cuda")
    A32 = torch.empty(64, device="cuda")
    f = torch.empty(lib.mpdok_lu_factor_size(8, N.F16), dtype=torch.uint8, device="cuda")
    w = torch.empty(lib.mpdok_lu_work_size(8, N.F16), dtype=torch.uint8, device="cuda")
    assert lib.mpdok_lu_factor_copy(ptr(A), 8, 8, N.F16, 0, ptr(f), f.numel(), ptr(w), w.numel(), ptr(A32), 7,
                                    stream_handle()) < 0
