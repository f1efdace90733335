"""GPU: one Arnoldi cycle of the fused step against FP64 least squares over the same Krylov space."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _optimal_residual(A, b, m):
    """min ||b - A V y|| / ||b|| over the m-dimensional Krylov space (FP64 Arnoldi, two passes)."""
    n = len(b)
    V = np.zeros((n, m + 1))
    H = np.zeros((m + 1, m))
    V[:, 0] = b / np.linalg.norm(b)
    for k in range(m):
        w = A @ V[:, k]
        for _ in range(2):
            h = V[:, :k + 1].T @ w
            w -= V[:, :k + 1] @ h
            H[:k + 1, k] += h
        H[k + 1, k] = np.linalg.norm(w)
        if H[k + 1, k] < 1e-14:
            break
        V[:, k + 1] = w / H[k + 1, k]
    e = np.zeros(m + 1)
    e[0] = 1.0
    y = np.linalg.lstsq(H, e, rcond=None)[0]
    return np.linalg.norm(b / np.linalg.norm(b) - A @ (V[:, :m] @ y))


@pytest.mark.parametrize("passes", [1, 2])
@pytest.mark.parametrize("n,m", [(1, 1), (63, 3), (64, 4), (65, 5), (513, 31), (700, 33), (4200, 40), (9000, 8)])
def test_one_cycle_reaches_the_optimal_residual(n, m, passes):
    """Sizes around the rows per CTA (64, above 4096 more), four-column groups,
    32-column sums and 32-entry scans.  The FP32 basis and operator are off by
    a few 2^-24 per step: sqrt(m) times a factor of 50 for the condition number."""
    from mpdok_gb300.dense_krylov import DenseLinearOperator, gmres
    from mpdok_gb300.solvers import MixedSolver
    rng = np.random.default_rng(n + m)
    A = np.diag(np.linspace(1.0, 50.0, n)) + rng.standard_normal((n, n)) * (0.3 / np.sqrt(n))
    b = rng.standard_normal(n)
    if passes == 2:
        _, info = MixedSolver(method="gmres-ir", restart=m, maxiter_outer=1).solve(A, b, tol=1e-30)
        rel = info["history"][-1][1]
    else:
        _, h, _ = gmres(DenseLinearOperator(A, verbose=False), b, tol=1e-30, maxiter=m, restart=m)
        rel = h[-1][1]
    ref = _optimal_residual(A, b, m)
    assert abs(rel - ref) <= 50 * np.sqrt(m) * 2.0 ** -24
