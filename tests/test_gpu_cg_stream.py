"""GPU: CG streams a matrix larger than the caches through shared memory that is refilled as
soon as it has been read.  A refill that overtakes a read shows as different bits; one was once
seen in some 10^8 units of 4 KB, so a thousand million of them are run."""
import torch
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,bsz", [(15000, 256), (11000, 128)])
def test_same_bits_over_many_units(hs, ctx, N, bsz):
    g = torch.Generator(device="cuda")
    g.manual_seed(N)
    X = torch.rand((N, 16), dtype=torch.float64, device="cuda", generator=g)
    ctx.set_problem(N, bsz)
    A = hs.SymmetricMatrix(N, bsz, device="cuda:0")
    hs.MatrixGenerator.assemble(ctx, A.matrixData, X, 1.0, 1.0, 1e-4)
    b = hs.RightHandSide(N, bsz, device="cuda:0")
    b.rightHandSideData[:N] = torch.randn(N, dtype=torch.float64, device="cuda", generator=g)
    units = A.matrixData.numel() // 512
    iterations = min(1000, 10 ** 8 // units)
    first = hs.CG(A, b, ctx).solveHeterogeneous(epsilon=0.0, iMax=iterations)
    for _ in range(10 ** 9 // 2 // (units * iterations)):
        again = hs.CG(A, b, ctx).solveHeterogeneous(epsilon=0.0, iMax=iterations)
        assert torch.equal(first.x, again.x)
