"""GPU: CG on the device against the launch-per-operation driver in the reference's order, on an
ill-conditioned system that takes over a thousand iterations and several launches."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_agrees_with_the_reference_order(hs, ctx):
    """Both end with ||b - K x|| <= 2 eps ||b||, so they differ by at most 4 eps ||b|| ||K^-1||,
    and ||K^-1|| <= 1 / sn2."""
    N, bsz, sn2, eps = 3000, 128, 2e-4, 1e-8
    g = torch.Generator(device="cuda")
    g.manual_seed(N + bsz)
    X = torch.rand((N, 8), dtype=torch.float64, device="cuda", generator=g)
    ctx.set_problem(N, bsz)
    A = hs.SymmetricMatrix(N, bsz, device="cuda:0")
    hs.MatrixGenerator.assemble(ctx, A.matrixData, X, 0.5, 1.0, sn2)
    b = hs.RightHandSide(N, bsz, device="cuda:0")
    b.rightHandSideData[:N] = torch.sin(X.sum(dim=1)) + 0.1 * torch.randn(N, dtype=torch.float64, device="cuda",
                                                                           generator=g)
    here = hs.CG(A, b, ctx).solveHeterogeneous(epsilon=eps, iMax=20000)
    ctx.set_reference_order(8)
    try:
        there = hs.CG(A, b, ctx).solveHeterogeneous(epsilon=eps, iMax=20000)
    finally:
        ctx.set_reference_order(0)
    assert here.iterations > 1000 and there.iterations > 1000
    norm = torch.linalg.norm(b.rightHandSideData).item()
    assert torch.linalg.norm(here.x - there.x).item() <= 4 * eps * norm / sn2
