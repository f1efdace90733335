"""GPU: the zero pivots that the clustered panel factorization reports, against an FP64 LU on the CPU."""
import numpy as np
import pytest
import scipy.linalg
import torch

pytestmark = pytest.mark.gpu


def _equilibrated(A, lu):
    _, _, _, dr, dc = lu.export()
    return dr.double().cpu().numpy()[:, None] * A * dc.double().cpu().numpy()[None, :]


@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, 384, 385, 768, 770, 1537, 3073])
@pytest.mark.parametrize("kind", ["normal", "signs"])
def test_regular_matrices_report_none(n, kind):
    """N(0, 1) matrices, and ones of -1, 0 and 1 plus 1e-3 of noise: with pivots above
    1e-4 (FP64, checked here; FP32 factors are off by some n 2^-24) info is 0."""
    from mpdok_gb300.lu import LUFactorization
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n))
    if kind == "signs":
        A = rng.integers(-1, 2, (n, n)) + 1e-3 * A + 0.5 * np.eye(n)
    lu = LUFactorization(torch.from_numpy(A).cuda(), dtype="fp32", pivoting=True)
    pivots = np.abs(np.diag(scipy.linalg.lu_factor(_equilibrated(A, lu))[0]))
    assert pivots.min() > 1e-4
    assert lu.info == 0


@pytest.mark.parametrize("n,col", [(1, 0), (40, 0), (40, 39), (200, 31), (200, 32), (200, 150), (900, 127), (900, 128),
                                   (3100, 1000), (3100, 3099)])
def test_the_first_zero_pivot_is_reported(n, col):
    """A column of zeros stays one under every exchange and update: its pivot is the first that is zero."""
    from mpdok_gb300.lu import LUFactorization
    rng = np.random.default_rng(n + col)
    A = rng.standard_normal((n, n))
    A[:, col] = 0.0
    lu = LUFactorization(torch.from_numpy(A).cuda(), dtype="fp32", pivoting=True)
    assert lu.info == col + 1
