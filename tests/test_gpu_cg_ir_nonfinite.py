"""GPU: a NaN in the matrix ends the multi-column CG-IR with a status, not as converged."""
import numpy as np
import pytest
import torch

from oracle import krylov_ref as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precond", [False, True])
@pytest.mark.parametrize("k", [1, 3])
def test_nan_matrix_is_reported(k, precond):
    from mpdok_gb300 import _native as N
    from mpdok_gb300.batch import CholeskyPreconditioner
    from mpdok_gb300.dense_krylov import DenseLinearOperator, cg_ir
    rng = np.random.default_rng(k)
    C = rng.uniform(0, 1, (200, 2))
    A = O.rbf_matrix(C, gamma=100.0, reg=1e-1)
    B = torch.from_numpy(rng.standard_normal((200, k))).cuda()
    pc = CholeskyPreconditioner(C, 10.0, 1e-1, nrhs=k) if precond else None
    x, _, converged = cg_ir(DenseLinearOperator(torch.from_numpy(A).cuda(), verbose=False), B, precond=pc, tol=1e-11)
    assert converged
    A[17, 3] = np.nan
    with pytest.raises(N.MPDOKError, match="non-finite residual") as e:
        cg_ir(DenseLinearOperator(torch.from_numpy(A).cuda(), verbose=False), B, precond=pc, tol=1e-11)
    assert e.value.status == N.ERR_NONFINITE
