"""GPU suite: the persistent CG at the edges of its division of the matrix (fewer units than
warps, ranges that stay in shared memory, ranges that cross several block columns, padding),
several launches of one solve, and the loop's end conditions."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _problem(hs, ctx, N, bsz, sn2=1e-2):
    g = torch.Generator(device="cuda")
    g.manual_seed(N + bsz)
    X = torch.rand((N, 8), dtype=torch.float64, device="cuda", generator=g)
    y = torch.sin(X.sum(dim=1)) + 0.1 * torch.randn(N, dtype=torch.float64, device="cuda", generator=g)
    ctx.set_problem(N, bsz)
    A = hs.SymmetricMatrix(N, bsz, device="cuda:0")
    hs.MatrixGenerator.assemble(ctx, A.matrixData, X, 0.5, 1.0, sn2)
    b = hs.RightHandSide(N, bsz, device="cuda:0")
    b.rightHandSideData[:N] = y
    K = torch.exp(-2.0 * torch.cdist(X, X, compute_mode="donot_use_mm_for_euclid_dist").square())
    K.diagonal().add_(sn2)
    return A, b, K, y


@pytest.mark.parametrize("bsz,N", [(128, n) for n in (1, 100, 128, 129, 700, 2600, 5000)] +
                         [(256, n) for n in (1, 200, 257, 1000, 2600, 5000, 9001)])
def test_converges_to_the_tolerance(hs, ctx, bsz, N):
    """||b - K x|| <= 2 eps ||b|| at the end (the recurrence's residual meets eps; the true
    one is recomputed every 50 iterations), the same bits every time, zero padding."""
    A, b, K, y = _problem(hs, ctx, N, bsz)
    cg = hs.CG(A, b, ctx).solveHeterogeneous(epsilon=1e-9, iMax=5000)
    again = hs.CG(A, b, ctx).solveHeterogeneous(epsilon=1e-9, iMax=5000)
    assert torch.equal(cg.x, again.x) and cg.iterations == again.iterations
    assert not cg.x[N:].any()
    r = torch.linalg.norm(K @ cg.x[:N].cuda() - y)
    assert r <= 2e-9 * torch.linalg.norm(y)
    assert 0 < cg.iterations < 5000
    assert cg.delta_new <= 1e-18 * cg.delta_zero
    assert abs(cg.delta_zero - float(y @ y)) <= 1e-12 * float(y @ y)


def test_iteration_limit_and_zero_rhs(hs, ctx):
    A, b, K, y = _problem(hs, ctx, 1500, 128)
    short = hs.CG(A, b, ctx).solveHeterogeneous(epsilon=1e-12, iMax=7)
    assert short.iterations == 7 and short.delta_new > 1e-24 * short.delta_zero
    none = hs.CG(A, b, ctx).solveHeterogeneous(epsilon=1e-12, iMax=0)
    assert none.iterations == 0 and not none.x.any()
    b.rightHandSideData.zero_()
    zero = hs.CG(A, b, ctx).solveHeterogeneous(epsilon=1e-12, iMax=100)
    assert zero.iterations == 0 and not zero.x.any()


def test_more_iterations_than_one_launch_runs(hs, ctx):
    """An ill-conditioned system needs over a thousand iterations, several launches; the
    result agrees with the launch-per-operation path in the reference's order (both within
    eps cond of the solution)."""
    A, b, K, y = _problem(hs, ctx, 3000, 128, sn2=2e-4)
    cg = hs.CG(A, b, ctx).solveHeterogeneous(epsilon=1e-8, iMax=20000)
    assert cg.iterations > 1000
    r = torch.linalg.norm(K @ cg.x[:3000].cuda() - y)
    assert r <= 2e-8 * torch.linalg.norm(y)
