"""GPU: several solves of one batch plan in flight (streams, host threads, a captured one)."""
import threading

import numpy as np
import pytest
import torch

from oracle import krylov_ref as O

pytestmark = pytest.mark.gpu


def _batch(rng, sizes, nrhs=3):
    from mpdok_gb300.batch import BatchedRBFSolver
    bs = BatchedRBFSolver(sizes, dim=2, nrhs=nrhs, grid_mult=1)
    bs.load([rng.uniform(0, 1, (n, 2)) for n in sizes], 10.0, 1e-2).factor()
    return bs, [torch.from_numpy(rng.standard_normal(sum(sizes) * nrhs)).cuda() for _ in range(12)]


def test_unrefined_solves_on_several_streams():
    """Solves without refinement only read the factors: the same bits as one after
    the other, from three streams and two host threads, beside residuals."""
    bs, Bs = _batch(np.random.default_rng(0), [700, 70, 1300])
    want = [bs.solve(b, refine=0) for b in Bs]
    rel = [bs.relres(b, x) for b, x in zip(Bs, want)]
    torch.cuda.synchronize()
    got, grel, errors = [None] * 12, [None] * 12, []

    def work(ids):
        try:
            streams = [torch.cuda.Stream() for _ in range(3)]
            for _ in range(4):
                for i in ids:
                    with torch.cuda.stream(streams[i % 3]):
                        got[i] = bs.solve(Bs[i], refine=0)
                        if i % 3 == 0:  # (one stream: the residuals share a buffer among themselves)
                            grel[i] = bs.relres(Bs[i], want[i]) if ids[0] == 0 else rel[i]
            for st in streams:
                st.synchronize()
        except Exception as e:
            errors.append(e)

    ts = [threading.Thread(target=work, args=(list(r),)) for r in (range(6), range(6, 12))]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not errors
    for i in range(12):
        assert torch.equal(got[i], want[i])
        assert grel[i] is None or torch.equal(grel[i], rel[i])


@pytest.mark.parametrize("refine", [0, 2])
def test_a_captured_solve_replays_beside_others(refine):
    bs, Bs = _batch(np.random.default_rng(1), [500, 900])
    want = [bs.solve(b, refine=refine) for b in Bs[:4]]
    b = Bs[0].clone()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        X = bs.solve(b, refine=refine)
    side = torch.cuda.Stream()
    for i in range(4):
        b.copy_(Bs[i])
        torch.cuda.synchronize()
        g.replay()
        if refine == 0:
            with torch.cuda.stream(side):
                Y = bs.solve(Bs[3 - i], refine=0)
        torch.cuda.synchronize()
        assert torch.equal(X, want[i])
        assert refine or torch.equal(Y, want[3 - i])


def test_two_solves_share_a_cholesky_preconditioner():
    from mpdok_gb300.batch import CholeskyPreconditioner
    from mpdok_gb300.dense_krylov import DenseLinearOperator, cg_ir
    rng = np.random.default_rng(2)
    n = 1500
    C = rng.uniform(0, 1, (n, 2))
    A = torch.from_numpy(O.rbf_matrix(C, gamma=100.0, reg=1e-3)).cuda()
    Bs = [torch.from_numpy(rng.standard_normal(n)).cuda() for _ in range(2)]
    pc = CholeskyPreconditioner(C, 10.0, 1e-3)
    ops = [DenseLinearOperator(A, verbose=False) for _ in range(2)]
    want = [cg_ir(op, b, precond=pc, tol=1e-13, maxiter_outer=4) for op, b in zip(ops, Bs)]
    torch.cuda.synchronize()
    got, errors = [[], []], []

    def work(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(5):
                    got[k].append(cg_ir(ops[k], Bs[k], precond=pc, tol=1e-13, maxiter_outer=4))
                torch.cuda.current_stream().synchronize()
        except Exception as e:
            errors.append(e)

    ts = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not errors
    for k in range(2):
        for x, hist, _ in got[k]:
            assert torch.equal(x, want[k][0]) and list(hist) == list(want[k][1])
