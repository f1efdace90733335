"""Matrix-vector products whose columns start off the 16-byte vectors.

Such a product reads scalars, 256 rows apart per thread instead of consecutive
ones, but every row still sums the same terms in the same order: it has to give
the bits of the same matrix stored with aligned columns.
"""
import pytest
import torch

from mpdok_gb300 import _native as N

pytestmark = pytest.mark.gpu

DTYPES = [(torch.float64, 0), (torch.float32, 1), (torch.bfloat16, 2), (torch.float16, 3)]


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (255, 3, 1), (1025, 515, 2), (2047, 700, 1),
                                   (2049, 4097, 8), (5003, 5003, 1), (1031, 129, 3)])
@pytest.mark.parametrize("dtype,code", DTYPES)
def test_misaligned_columns_same_bits(dtype, code, m, n, k):
    from mpdok_gb300._device import ptr, stream_handle
    lib = N.load()
    g = torch.Generator("cpu").manual_seed(m + 7 * n)
    acc = torch.float64 if code == 0 else torch.float32
    M = torch.randn(n, m, generator=g, dtype=torch.float64).to(dtype)
    X = torch.randn(k, n, generator=g, dtype=torch.float64).to(acc).cuda()
    out = []
    for lda in ((m + 15) // 16 * 16, (m + 15) // 16 * 16 + 1):
        A = torch.zeros(n, lda, dtype=dtype)
        A[:, :m] = M
        A = A.cuda()
        w = torch.empty(lib.mpdok_gemv_workspace_size(code, m, n, k, 0), dtype=torch.uint8, device="cuda")
        Y = torch.full((k, m), float("nan"), dtype=acc, device="cuda")
        N.check(lib.mpdok_gemv(code, 0, ptr(A), lda, m, n, ptr(X), n, k, ptr(Y), m, 1.0, 0.0,
                               ptr(w), w.numel(), stream_handle()))
        out.append(Y.cpu())
    assert torch.equal(out[0], out[1])
