"""GPU: FP64 kernel entries (integer-pipe exponential, mirrored tiles) against extended precision."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def _reference(R, C, gamma, kernel):
    R, C = R.astype(np.longdouble), C.astype(np.longdouble)
    d2 = ((R[:, None, :] - C[None, :, :]) ** 2).sum(-1)
    t = np.longdouble(gamma) * d2
    return (np.exp(-t) if kernel == "gaussian" else np.sqrt(1 + t)), t


def _check(A, ref, t):
    """d2 is formed in FP64 with at most 2 D roundings (D <= 3), which the exponential
    turns into 6 u t; the exponential itself is within 1.1 ulp up to t = 200
    and 3.2 ulp beyond; sqrt is correctly rounded (half its argument's error)."""
    tol = (6 * t + 8) * U
    err = np.abs(A.astype(np.longdouble) - ref)
    assert np.all(err <= tol * ref + 5e-324)


@pytest.mark.parametrize("kernel", ["gaussian", "mq"])
@pytest.mark.parametrize("dim", [1, 2, 3])
@pytest.mark.parametrize("n,pad", [(1, 0), (63, 1), (64, 0), (65, 2), (200, 0)])
def test_square_fp64_assembly(n, pad, dim, kernel):
    from mpdok_gb300._device import fortran_empty
    from mpdok_gb300.rbf_kernel import assemble
    rng = np.random.default_rng(n + dim)
    X = rng.uniform(-1, 2, (n, dim))
    Xd = torch.from_numpy(X).cuda()
    gamma = 37.0
    full = fortran_empty(n + pad, n, torch.float64)
    full.fill_(7.0)
    out = full[:n]
    assemble(Xd, gamma=gamma, kernel=kernel, out=out)
    A = out.cpu().numpy()
    ref, t = _reference(X, X, gamma, kernel)
    _check(A, ref, t)
    assert np.array_equal(A, A.T) and np.all(full[n:].cpu().numpy() == 7.0)
    # the same entries as the general kernel, and the nugget on the diagonal only
    B = assemble(Xd, Xd.clone(), gamma=gamma, kernel=kernel).cpu().numpy()
    assert np.array_equal(A, B)
    D = assemble(Xd, gamma=gamma, reg=0.25, kernel=kernel).cpu().numpy()
    assert np.array_equal(D, A + 0.25 * np.eye(n))


@pytest.mark.parametrize("gamma", [0.0, -2.0, 1e-300, 3e-9, 1.0, 1e4, 1e6, 1e300])
def test_gaussian_over_the_range_of_gamma(gamma):
    """Results near 1, tiny, denormal, zero and above 1, and zero distances."""
    from mpdok_gb300.rbf_kernel import assemble
    rng = np.random.default_rng(3)
    R = np.concatenate([rng.uniform(0, 1, (40, 1)), np.linspace(0, 0.05, 40)[:, None], [[0.0], [5e-200]]])
    C = np.concatenate([rng.uniform(0, 1, (29, 1)), [[0.0]]])
    A = assemble(torch.from_numpy(R).cuda(), torch.from_numpy(C).cuda(), gamma=gamma).cpu().numpy()
    ref, t = _reference(R, C, gamma, "gaussian")
    tol = (6 * np.abs(t) + 8) * U
    normal = ref > 2.3e-308
    assert np.all(np.abs(A - ref)[normal] <= (tol * ref)[normal])
    assert np.all(np.abs(A - ref)[~normal] <= 2.3e-308 * 1e-12 + 5e-324)


@pytest.mark.parametrize("kernel", ["gaussian", "mq"])
@pytest.mark.parametrize("dim", [1, 2, 3])
@pytest.mark.parametrize("n,m,k", [(1, 1, 1), (127, 255, 2), (129, 257, 3), (300, 40, 8), (260, 300, 5)])
def test_fp64_evaluation(n, m, k, dim, kernel):
    from mpdok_gb300.matfree import rbf_evaluate
    rng = np.random.default_rng(n + m + k)
    C, Q, a = rng.uniform(0, 1, (n, dim)), rng.uniform(0, 1, (m, dim)), rng.standard_normal((n, k))
    out = rbf_evaluate(torch.from_numpy(a).cuda(), torch.from_numpy(C).cuda(), torch.from_numpy(Q).cuda(), gamma=20.0,
                       kernel=kernel).cpu().numpy()
    ref, t = _reference(Q, C, 20.0, kernel)
    exact = ref @ a.astype(np.longdouble)
    # entries within (6 t + 8) u, sums of n products within n u
    bound = ((ref * (6 * t + 8)) @ np.abs(a) + n * (np.abs(ref) @ np.abs(a))) * U
    assert np.all(np.abs(out - exact) <= bound)


@pytest.mark.parametrize("k", [1, 2, 3, 8])
@pytest.mark.parametrize("kernel", ["gaussian", "mq"])
def test_adjoint_contraction_for_each_column_count(k, kernel):
    """grad_coords, grad_eps and grad_reg of the batch contraction against dense
    FP64 formulas: sums of n k products of relative rounding a few u each."""
    from mpdok_gb300.batch import BatchedRBFSolver, pack_rhs
    rng = np.random.default_rng(k)
    sizes, dim, eps = [65, 130], 2, [3.0, 5.0]
    Cs = [rng.uniform(0, 1, (n, dim)) for n in sizes]
    Xs, Ls = ([rng.standard_normal((n, k)) for n in sizes] for _ in range(2))
    bs = BatchedRBFSolver(sizes, dim=dim, nrhs=k, kernel=kernel, grid_mult=1)
    bs.load(Cs, eps, 1e-2)
    gc, ge, gr = (t.cpu().numpy() for t in bs.adjoint(pack_rhs(Xs, k), pack_rhs(Ls, k)))
    o = 0
    for i, (C, X, L, n) in enumerate(zip(Cs, Xs, Ls, sizes)):
        df = C[:, None, :] - C[None, :, :]
        r2 = (df ** 2).sum(-1)
        g2 = eps[i] ** 2
        if kernel == "gaussian":
            phi = np.exp(-g2 * r2)
            g, h = -g2 * phi, -r2 * phi
        else:
            phi = np.sqrt(1 + g2 * r2)
            g, h = 0.5 * g2 / phi, 0.5 * r2 / phi
        u = L @ X.T
        w = u + u.T
        c_terms = -2.0 * (w * g)[:, :, None] * df
        tol = 1e-14 * n * k
        assert np.all(np.abs(gc[o:o + n] - c_terms.sum(1)) <= tol * np.abs(c_terms).sum(1).max())
        assert abs(ge[i] + 2 * eps[i] * (u * h).sum()) <= tol * 2 * eps[i] * np.abs(u * h).sum()
        assert abs(gr[i] + (L * X).sum()) <= tol * np.abs(L * X).sum()
        o += n
