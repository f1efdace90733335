"""GPU: a batch solve whose bounded wait runs out is reported (made by the host: the
first ticket is raised, so that no block ever solves block 0, and the wait limit
is shortened; every wait ends and the device stays usable)."""
import numpy as np
import pytest
import torch

from oracle import krylov_ref as O

pytestmark = pytest.mark.gpu


@pytest.fixture
def no_block_zero(native_lib):
    from mpdok_gb300 import _native as N
    def on():
        N.check(native_lib.mpdok_debug_set(1, 2000), "limit")
        N.check(native_lib.mpdok_debug_set(2, 1), "ticket")
    def off():
        N.check(native_lib.mpdok_debug_set(2, 0), "ticket")
        N.check(native_lib.mpdok_debug_set(1, 0), "limit")
    yield on, off
    off()


def _batch(rng, sizes=(200,), nrhs=2):
    from mpdok_gb300.batch import BatchedRBFSolver
    bs = BatchedRBFSolver(list(sizes), dim=2, nrhs=nrhs, grid_mult=1)
    Cs = [rng.uniform(0, 1, (n, 2)) for n in sizes]
    bs.load(Cs, 10.0, 1e-2).factor()
    return bs, Cs, torch.from_numpy(rng.standard_normal(sum(sizes) * nrhs)).cuda()


@pytest.mark.parametrize("later", ["dag_status", "load", "factor", "solve", "step", "relres", "adjoint", "perturbed_pivots",
                                   "run_graph"])
@pytest.mark.parametrize("refine", [0, 2])
def test_next_call_reports_it_once(no_block_zero, later, refine):
    on, off = no_block_zero
    bs, Cs, b = _batch(np.random.default_rng(0))
    good = bs.solve(b, refine=2)
    bs.build_graph(b, refine=2)
    on()
    X = bs.solve(b, refine=refine)
    torch.cuda.synchronize()
    off()
    assert torch.isnan(X).any()
    call = dict(dag_status=bs.dag_status, load=lambda: bs.load(Cs, 10.0, 1e-2), factor=bs.factor,
                solve=lambda: bs.solve(b), step=lambda: bs.step(b), relres=lambda: bs.relres(b, good),
                adjoint=lambda: bs.adjoint(good, good), perturbed_pivots=bs.perturbed_pivots,
                run_graph=bs.run_graph)[later]
    with pytest.raises(RuntimeError, match="ran out"):
        call()
    call()
    bs.factor()
    bs.dag_status()
    assert torch.equal(bs.solve(b, refine=2), good)


def test_a_training_step_reports_it(no_block_zero):
    from mpdok_gb300.batch import rbf_batch_solve
    on, off = no_block_zero
    bs, Cs, b = _batch(np.random.default_rng(1))
    C = torch.from_numpy(Cs[0]).cuda().requires_grad_(True)
    eps, reg = torch.tensor(10.0), torch.tensor(1e-2)
    X = rbf_batch_solve(C, eps, reg, b, bs)
    X.sum().backward()
    want = C.grad.clone()
    on()
    X = rbf_batch_solve(C, eps, reg, b, bs)
    torch.cuda.synchronize()
    off()
    with pytest.raises(RuntimeError, match="ran out"):
        X.sum().backward()
    C.grad = None
    rbf_batch_solve(C, eps, reg, b, bs).sum().backward()
    assert torch.equal(C.grad, want)


def test_the_cholesky_preconditioner_reports_it(no_block_zero):
    """... as a status of its own solve, and the next solve is normal."""
    from mpdok_gb300.batch import CholeskyPreconditioner
    from mpdok_gb300.dense_krylov import DenseLinearOperator, cg_ir
    on, off = no_block_zero
    rng = np.random.default_rng(2)
    C = rng.uniform(0, 1, (300, 2))
    A = torch.from_numpy(O.rbf_matrix(C, gamma=100.0, reg=1e-2)).cuda()
    b = torch.from_numpy(rng.standard_normal(300)).cuda()
    op = DenseLinearOperator(A, verbose=False)
    pc = CholeskyPreconditioner(C, 10.0, 1e-2)
    on()
    with pytest.raises(RuntimeError, match="ran out"):
        cg_ir(op, b, precond=pc, tol=1e-12)
    off()
    x, _, converged = cg_ir(op, b, precond=pc, tol=1e-12)
    assert converged and O.relres(A.cpu().numpy(), x.reshape(-1).cpu().numpy(), b.cpu().numpy()) < 1e-11
