"""GPU: many right-hand sides of a large system, where the residual runs on the tensor cores."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(2304, 11), (2304, 20), (4500, 200)])
def test_groups_take_the_steps_they_would_take_alone(n, k):
    """Bit-identical to one mpdok_lu_ir_solve_multi call per group: with a remainder
    below four columns (its residual is the FP64 product), with one of four, and
    with a second pass that needs more workspace than the first (n = 4500: 72
    columns after 128).  The bytes behind the workspace stay as they were."""
    from mpdok_gb300 import _native as N
    from mpdok_gb300._device import fortran_empty, ptr, stream_handle
    from mpdok_gb300.lu import LUFactorization
    from mpdok_gb300.rbf_kernel import build_rbf_kernel
    rng = np.random.default_rng(n + k)
    Ad, _ = build_rbf_kernel(torch.from_numpy(rng.uniform(0, 1, (n, 2))).cuda(), gamma=0.2 * n, reg=0.1)
    Bd = torch.from_numpy(rng.standard_normal((k, n))).cuda().t()
    lu = LUFactorization(Ad, dtype="fp32")
    lib = N.load()
    size = lib.mpdok_lu_ir_many_work_size(n, k)
    work = torch.full((size + (64 << 20),), 0x5a, dtype=torch.uint8, device="cuda")
    X = fortran_empty(n, k, torch.float64)
    infos = (N.SolveInfo * ((k + 7) // 8))()
    N.check(lib.mpdok_lu_ir_solve_many(ptr(Ad), n, n, ptr(lu.factors), lu.fdtype, k, ptr(Bd), n, ptr(X), n, 1e-12, 6,
                                       ptr(work), size, infos, stream_handle()), "many")
    assert torch.all(work[size:] == 0x5a)
    for q in range((k + 7) // 8):
        c, kk = 8 * q, min(8, k - 8 * q)
        Y = fortran_empty(n, kk, torch.float64)
        w = torch.empty(lib.mpdok_lu_ir_multi_work_size(n, kk), dtype=torch.uint8, device="cuda")
        one = N.SolveInfo()
        N.check(lib.mpdok_lu_ir_solve_multi(ptr(Ad), n, n, ptr(lu.factors), lu.fdtype, kk, ptr(Bd[:, c:c + kk]), n,
                                            ptr(Y), n, 1e-12, 6, ptr(w), w.numel(), ctypes.byref(one),
                                            stream_handle()), "multi")
        assert one.converged and infos[q].converged
        assert torch.equal(Y, X[:, c:c + kk])
        assert one.history_list() == infos[q].history_list()


def test_finished_groups_leave_the_residual():
    """Five groups, four of them zero and so done at once: the products after the
    first cover the fifth only (8 bytes n^2 + 16 bytes n per column that they
    multiply), and its steps are the ones it takes alone."""
    from mpdok_gb300 import _native as N
    from mpdok_gb300.lu import LUFactorization
    from mpdok_gb300.rbf_kernel import build_rbf_kernel
    n = 2304
    rng = np.random.default_rng(3)
    Ad, _ = build_rbf_kernel(torch.from_numpy(rng.uniform(0, 1, (n, 2))).cuda(), gamma=0.2 * n, reg=0.1)
    B = torch.zeros((40, n), dtype=torch.float64, device="cuda").t()
    B[:, 24:32] = torch.from_numpy(rng.standard_normal((n, 8))).cuda()
    lu = LUFactorization(Ad, dtype="fp16")
    Y, alone = lu.solve_ir_many(Ad, B[:, 24:32], tol=1e-12, maxiter_outer=10)
    N.profile_enable(True)
    try:
        X, info = lu.solve_ir_many(Ad, B, tol=1e-12, maxiter_outer=10)
        torch.cuda.synchronize()
        _, launches, work = N.profile_query(N.PROF_GEMV_F64)
    finally:
        N.profile_enable(False)
    assert info["converged"] and torch.equal(X[:, 24:32], Y) and info["history"][3] == alone["history"][0]
    assert torch.all(X[:, :24] == 0) and torch.all(X[:, 32:] == 0)
    assert launches == len(info["history"][3]) > 2
    assert work == launches * 8.0 * n * n + 16.0 * n * (40 + 8 * (launches - 1))
