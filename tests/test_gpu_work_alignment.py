"""GPU: work buffers that start on an 8-byte boundary only."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _system(n, k):
    rng = np.random.default_rng(n)
    C = torch.from_numpy(rng.uniform(0, 1, (n, 2))).cuda()
    from mpdok_gb300.rbf_kernel import build_rbf_kernel
    A, _ = build_rbf_kernel(C, gamma=0.2 * n, reg=0.1)
    return A, torch.from_numpy(rng.standard_normal((k, n))).cuda().t()


@pytest.mark.parametrize("n,k", [(300, 8), (2100, 8), (2100, 20)])
def test_many_right_hand_sides(n, k):
    from mpdok_gb300 import _native as N
    from mpdok_gb300._device import fortran_empty, ptr, stream_handle
    from mpdok_gb300.lu import LUFactorization
    A, B = _system(n, k)
    lu = LUFactorization(A, dtype="fp32")
    lib = N.load()
    size = lib.mpdok_lu_ir_many_work_size(n, k)
    work = torch.empty(size + 8, dtype=torch.uint8, device="cuda")[8:]
    assert work.data_ptr() % 16 == 8
    X = fortran_empty(n, k, torch.float64)
    infos = (N.SolveInfo * ((k + 7) // 8))()
    N.check(lib.mpdok_lu_ir_solve_many(ptr(A), n, n, ptr(lu.factors), lu.fdtype, k, ptr(B), n, ptr(X), n, 1e-12, 6,
                                       ptr(work), size, infos, stream_handle()), "many")
    assert all(i.converged for i in infos)
    assert ((B - A @ X).norm(dim=0) / B.norm(dim=0)).max().item() <= 2e-12


@pytest.mark.parametrize("n", [100, 700])
def test_pivoted_fp32_factorization(n):
    """The same factors as with an aligned buffer."""
    from mpdok_gb300 import _native as N
    from mpdok_gb300._device import ptr, stream_handle
    A, _ = _system(n, 1)
    lib = N.load()
    size = lib.mpdok_lu_work_size(n, N.F32)
    facs = []
    for off in (0, 8):
        fac = torch.zeros(lib.mpdok_lu_factor_size(n, N.F32), dtype=torch.uint8, device="cuda")
        work = torch.zeros(size + off, dtype=torch.uint8, device="cuda")[off:]
        st = lib.mpdok_lu_factor(ptr(A), n, n, N.F32, 1, ptr(fac), fac.numel(), ptr(work), size, stream_handle())
        assert st == 0, N.last_error()
        facs.append(fac)
    assert torch.equal(*facs)
