"""GPU: the pivoted panel factorization inside one cluster (panels of up to 6144 rows)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["normal", "ties"])
@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, 384, 385, 768, 770, 1537, 3073, 6145])
def test_pivoted_factors_at_the_cluster_sizes(n, kind):
    """Sizes around the sub-panels (32), the panels (128), the rows per CTA (384)
    and the cluster sizes 1, 2, 4, 8, 16; 6145 starts on the taller-panel
    kernel.  |L| <= 1 (each pivot is the largest of its column) and, to FP32
    rounding, P Dr A Dc = L U: 8 x 2^-24 of |L| |U| in the Frobenius norm."""
    from mpdok_gb300.lu import LUFactorization
    g = torch.Generator("cuda").manual_seed(n)
    A = torch.randn(n, n, device="cuda", dtype=torch.float64, generator=g)
    if kind == "ties":  # many equal magnitudes, a zero diagonal
        A = torch.randint(-1, 2, (n, n), device="cuda", generator=g).double()
        A.diagonal().zero_()
        A += 1e-3 * torch.randn(n, n, device="cuda", dtype=torch.float64, generator=g).round(decimals=1)
    lu = LUFactorization(A, dtype="fp32", pivoting=True)
    LU, ipiv, perm, dr, dc = lu.export()
    if lu.info:
        return  # (singular draws of the smallest sizes: LAPACK's info is tested elsewhere)
    p = torch.arange(n)
    for i, r in enumerate(ipiv.tolist()):
        assert i <= r < n
        p[i], p[r] = p[r].clone(), p[i].clone()
    assert torch.equal(p, perm.cpu().long())
    LU = LU.double()
    L, U = torch.tril(LU, -1), torch.triu(LU)
    assert L.abs().max().item() <= 1.0 + 2.0 ** -23 if n > 1 else True
    L.diagonal().fill_(1.0)
    W = (dr.double()[:, None] * A * dc.double()[None, :])[perm.long()]
    assert (L @ U - W).norm() <= 8 * 2.0 ** -24 * (L.abs() @ U.abs()).norm()


def test_zero_column_is_reported_and_left():
    from mpdok_gb300.lu import LUFactorization
    g = torch.Generator("cuda").manual_seed(1)
    A = torch.randn(900, 900, device="cuda", dtype=torch.float64, generator=g)
    A[:, 300] = 0.0
    lu = LUFactorization(A, dtype="fp32", pivoting=True)
    assert lu.info == 301
    LU, ipiv, *_ = lu.export()
    assert ipiv[300].item() == 300 and torch.all(LU[:, 300] == 0)
