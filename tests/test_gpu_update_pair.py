"""The far update on CTA pairs (two SMs per 256 x 256 tile) against FP64.

Sizes past its rule (K >= 2048 and two 128 x 256 tiles per SM) with the edges
where it can go wrong: two row blocks only, an odd number of row blocks (the
last pair's second CTA holds none), rows and columns that end inside a warp's
32 rows, a 16-column chunk or the second CTA's half of B.
"""
import pytest
import torch

from mpdok_gb300 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(129, 39000, 2048), (2305, 4353, 2048), (4096, 2560, 2112), (2689, 4225, 2048),
                                   (4481, 2305, 4096), (12545, 3073, 2048)])
@pytest.mark.parametrize("dtype,code", [(torch.float16, N.F16), (torch.bfloat16, N.BF16)])
def test_pair_update(dtype, code, m, n, k):
    from mpdok_gb300._device import ptr, stream_handle
    lib = N.load()
    g = torch.Generator("cuda").manual_seed(m + n)
    A = torch.randn(m, k, generator=g, device="cuda").to(dtype)
    B = torch.randn(n, k, generator=g, device="cuda").to(dtype)
    ldc = (m + 3) // 4 * 4 + 4
    C0 = torch.randn(n, ldc, generator=g, device="cuda")
    C = C0.clone()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    N.check(lib.mpdok_gemm_update(ptr(C), ldc, ptr(A), ptr(B), m, n, k, code, N.ENGINE_TENSOR, ptr(err),
                                  stream_handle()))
    assert err.item() == 0
    assert torch.equal(C[:, m:], C0[:, m:])
    A, B = A.double(), B.double()
    for j in range(0, n, 4096):
        e = slice(j, min(n, j + 4096))
        ref = C0[e, :m].double() - B[e] @ A.T
        # one truncation (2^-23) of the running sum per 16 products and 16
        # inside each, then one rounding of the subtraction
        bound = (k / 16 + 16) * 2.0 ** -23 * (B[e].abs() @ A.abs().T) + 2.0 ** -23 * (ref.abs() + C0[e, :m].abs())
        assert ((C[e, :m].double() - ref).abs() <= bound).all()
