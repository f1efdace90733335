"""GPU: batched solves at the edges of the 64-row blocks and the four-column groups."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 63, 64, 65, 127, 128, 129, 200, 257]


@pytest.mark.parametrize("arith", ["f64", "df32"])
@pytest.mark.parametrize("nrhs", [1, 3, 4, 5, 8])
def test_solves_at_block_and_group_edges(arith, nrhs):
    """Against dense FP64 solves: kappa <= 1e4 here, so two refined solves agree
    to kappa 2^-53 times the usual n: 1e-9.  The task graph gives the same bits."""
    from mpdok_gb300.batch import BatchedRBFSolver, unpack_rhs
    rng = np.random.default_rng(nrhs)
    Xs = [rng.uniform(0, 1, (n, 2)) for n in SIZES]
    Bs = [rng.standard_normal((n, nrhs)) for n in SIZES]
    eps = np.linspace(3.0, 8.0, len(SIZES))
    bs = BatchedRBFSolver(SIZES, dim=2, nrhs=nrhs, arith=arith, grid_mult=1)
    bs.load(Xs, eps, 1e-1)
    X = bs.step(Bs, refine=2)
    bs.dag_status()
    for x, C, B, e in zip(unpack_rhs(X, SIZES, nrhs), Xs, Bs, eps):
        A = np.exp(-e * e * ((C[:, None] - C[None]) ** 2).sum(-1)) + 0.1 * np.eye(len(C))
        ref = np.linalg.solve(A, B)
        assert np.linalg.norm(x.cpu().numpy() - ref) <= 1e-9 * np.linalg.norm(ref)
    assert bs.perturbed_pivots() == 0
    bs.configure("dag:3")
    assert torch.equal(bs.step(Bs, refine=2), X)
    bs.dag_status()


def test_solve_without_refinement_and_a_graph_of_the_chain_solves():
    from mpdok_gb300.batch import BatchedRBFSolver, pack_rhs
    rng = np.random.default_rng(7)
    bs = BatchedRBFSolver(SIZES, dim=3, nrhs=6, grid_mult=1)
    bs.load([rng.uniform(0, 1, (n, 3)) for n in SIZES], 4.0, 1e-2).factor()
    B = pack_rhs([rng.standard_normal((n, 6)) for n in SIZES], 6)
    X = bs.solve(B, refine=0)
    assert bs.relres(B, X).max().item() < 1e-10  # double-float factor: 2^-48 times kappa
    Bb, Xb = bs.build_graph(B, refine=1)
    for _ in range(3):
        bs.run_graph()
    torch.cuda.synchronize()
    assert torch.equal(Xb, bs.solve(B, refine=1))


def test_indefinite_pivots_are_perturbed_and_counted():
    from mpdok_gb300.batch import BatchedRBFSolver
    C = np.zeros((70, 2))  # coincident centres: A = ones, every pivot but the first is zero
    bs = BatchedRBFSolver([70], dim=2, nrhs=1, grid_mult=1)
    bs.load([C], 1.0, 0.0).factor()
    assert bs.perturbed_pivots() == 69
