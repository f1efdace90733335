"""GPU: the triangular solves on systems whose last 128-row block and last 8-row vector are ragged."""
import numpy as np
import pytest
import torch
from scipy.linalg import solve_triangular

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,u", [("fp32", 2.0 ** -24), ("fp16", 2.0 ** -11), ("bf16", 2.0 ** -8)])
@pytest.mark.parametrize("n,k", [(129, 1), (257, 8), (300, 3), (511, 2), (520, 8)])
def test_ragged_blocks_match_the_exported_factors(dtype, u, n, k):
    """apply() and the multi-column solve against FP64 solves with the exported
    factors.  The off-diagonal part has norm 1/2, so every misread tile shows in
    the first digit.  The exported diagonal blocks are rounded to the factor
    type while the solves use FP32 ones: 4 u; FP32 sums of n terms: n 2^-24."""
    from mpdok_gb300.lu import LUFactorization
    rng = np.random.default_rng(n + k)
    A = np.eye(n) + rng.standard_normal((n, n)) * (0.25 / np.sqrt(n))
    lu = LUFactorization(A, dtype=dtype)
    assert lu.n_perturbed == 0
    LU, _, perm, dr, dc = (t.double().cpu().numpy() for t in lu.export())
    V = rng.standard_normal((n, k))

    def solve(v):
        y = solve_triangular(LU, (dr * v)[perm.astype(int)], lower=True, unit_diagonal=True)
        return dc * solve_triangular(LU, y, lower=False)

    tol = 4 * u + n * 2.0 ** -24
    for j in range(k):
        z = lu.apply(torch.from_numpy(V[:, j]).cuda()).double().cpu().numpy()
        ref = solve(V[:, j])
        assert np.linalg.norm(z - ref) <= tol * np.linalg.norm(ref)
    # one multi-column sweep and no refinement: X = LU^-1 B rounded to FP32
    X, _ = lu.solve_ir_many(torch.from_numpy(A).cuda(), torch.from_numpy(V).cuda(), tol=1e30, maxiter_outer=0)
    for j in range(k):
        ref = solve(V[:, j])
        assert np.linalg.norm(X[:, j].cpu().numpy() - ref) <= tol * np.linalg.norm(ref)
