"""Power-of-two equilibration of the pivoted LU by exponent arithmetic: scales and scaled entries, bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _scale(m):
    e = np.clip(np.frexp(m)[1], -120, 120)
    return np.where((m > 0) & np.isfinite(m), np.ldexp(1.0, -e), 1.0)


@pytest.mark.parametrize("n", [1, 3, 64, 255, 257, 700])
@pytest.mark.parametrize("spread", [20, 180])
def test_scales_and_entries(n, spread):
    """An upper triangular matrix keeps its rows and its multipliers are zero, so
    while its scaled entries and pivots stay finite and normal in FP32 its factors
    are the scaled matrix itself.  Rows and columns range over 2^+-spread, past
    the 2^120 clamp of the row scales; some entries are zero or subnormal."""
    from mpdok_gb300.lu import LUFactorization
    rng = np.random.default_rng(n + spread)
    A = rng.uniform(0.5, 1.0, (n, n)) * rng.choice([-1.0, 1.0], (n, n))
    A = np.ldexp(A, rng.integers(-spread, spread + 1, (n, 1)) + rng.integers(-20, 21, (1, n)))
    off = (rng.random((n, n)) < 0.1) & ~np.eye(n, dtype=bool)
    A = np.triu(np.where(off, rng.choice([0.0, 5e-320, -3e-310], (n, n)), A))
    LU, _, perm, dr, dc = LUFactorization(torch.from_numpy(A).cuda(), dtype="fp32", pivoting=True).export()
    r = _scale(np.abs(A).max(1))
    c = _scale((np.abs(A) * r[:, None]).max(0))
    assert np.array_equal(dr.cpu().numpy().astype(np.float64), r)
    assert np.array_equal(dc.cpu().numpy().astype(np.float64), c)
    assert np.array_equal(perm.cpu().numpy(), np.arange(n))
    assert np.array_equal(LU.cpu().numpy(), (A * r[:, None] * c[None, :]).astype(np.float32))
