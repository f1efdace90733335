"""GPU: many right-hand sides in groups of eight against the groups one by one."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fdtype", ["fp32", "fp16"])
@pytest.mark.parametrize("n,k", [(300, 1), (300, 8), (641, 9), (1000, 24), (500, 131), (200, 140)])
def test_groups_take_the_steps_they_would_take_alone(fdtype, n, k):
    """Bit-identical to one mpdok_lu_ir_solve_multi call per group, also when the
    groups stop at different steps (columns of one group are scaled solutions of
    a few eigenvectors, those of others white noise), with a remainder group
    and with more than 16 groups."""
    from mpdok_gb300 import _native as N
    from mpdok_gb300._device import fortran_empty, ptr, stream_handle
    from mpdok_gb300.lu import LUFactorization
    rng = np.random.default_rng(n + k)
    C = rng.uniform(0, 1, (n, 2))
    A = np.exp(-1600.0 * ((C[:, None] - C[None]) ** 2).sum(-1)) + 0.1 * np.eye(n)
    B = rng.standard_normal((n, k))
    B[:, :8] = 0.0
    B[0, :8] = 1.0
    Ad, Bd = torch.from_numpy(A).cuda(), torch.from_numpy(np.asfortranarray(B)).cuda()
    lu = LUFactorization(Ad, dtype=fdtype)
    X, info = lu.solve_ir_many(Ad, Bd, tol=1e-12, maxiter_outer=10)
    assert info["converged"] and len(info["history"]) == (k + 7) // 8
    lib = N.load()
    for q in range((k + 7) // 8):
        c, kk = 8 * q, min(8, k - 8 * q)
        Y = fortran_empty(n, kk, torch.float64)
        w = torch.empty(lib.mpdok_lu_ir_multi_work_size(n, kk), dtype=torch.uint8, device="cuda")
        one = N.SolveInfo()
        N.check(lib.mpdok_lu_ir_solve_multi(ptr(Ad), n, n, ptr(lu.factors), lu.fdtype, kk, ptr(Bd[:, c:c + kk]), n,
                                            ptr(Y), n, 1e-12, 10, ptr(w), w.numel(), ctypes.byref(one),
                                            stream_handle()), "multi")
        assert torch.equal(Y, X[:, c:c + kk])
        assert one.history_list() == info["history"][q]
