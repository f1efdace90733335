"""GPU: FP32 factors through the tensor-core update (three BF16 planes) keep FP32's accuracy."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pivoting", [False, True])
@pytest.mark.parametrize("n", [130, 257, 384, 641, 1153, 2200])
def test_fp32_factors_reproduce_the_matrix_to_fp32_rounding(n, pivoting):
    """Sizes around the 128-row panels, the 256-column tiles and the 1024-column
    super-panels, entries over many binades.  W, L and U are each rounded to
    FP32 and the sums of an entry's update add roundings of about one unit per
    block, all relative to |L| |U|: 8 x 2^-24 of it in the Frobenius norm.
    Dropping a plane of the operands would leave 2^-17."""
    from mpdok_gb300.lu import LUFactorization
    rng = np.random.default_rng(n)
    scale = 2.0 ** rng.integers(-10, 11, n)
    A = (np.eye(n) + rng.standard_normal((n, n)) * (0.25 / np.sqrt(n))) * scale[:, None] * scale[None, :]
    lu = LUFactorization(A, dtype="fp32", pivoting=pivoting)
    assert lu.n_perturbed == 0 and lu.info == 0
    LU, _, perm, dr, dc = (t.double().cpu().numpy() for t in lu.export())
    W = (dr[:, None] * A * dc[None, :])[perm.astype(int)]
    L, U = np.tril(LU, -1) + np.eye(n), np.triu(LU)
    assert np.linalg.norm(L @ U - W) <= 8 * 2.0 ** -24 * np.linalg.norm(np.abs(L) @ np.abs(U))
