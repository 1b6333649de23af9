"""GPU suite: the single-launch triangular sweeps at the edges of their division of labour:
the chain alone (1 to 3 block rows), one slice a CTA, several slices a CTA, padding in the
last block; FP64 factors and the mixed form's FP32 factor.  (The sizes also cross the
factor's switches between small and large update tiles and panel slabs.)"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _problem(hs, ctx, N, bsz):
    g = torch.Generator(device="cuda")
    g.manual_seed(N + bsz)
    X = torch.rand((N, 8), dtype=torch.float64, device="cuda", generator=g)
    y = torch.randn(N, dtype=torch.float64, device="cuda", generator=g)
    ctx.set_problem(N, bsz)
    A = hs.SymmetricMatrix(N, bsz, device="cuda:0")
    hs.MatrixGenerator.assemble(ctx, A.matrixData, X, 0.5, 1.0, 1e-2)
    K = torch.exp(-2.0 * torch.cdist(X, X, compute_mode="donot_use_mm_for_euclid_dist").square())
    K.diagonal().add_(1e-2)
    return A, K, y


SIZES = [(128, n) for n in (129, 256, 300, 640, 1000, 4777, 10001)] + [(256, n) for n in (257, 512, 700, 1300, 5000, 9001)]


@pytest.mark.parametrize("bsz,N", SIZES)
def test_fp64_sweeps(hs, ctx, bsz, N):
    """Backward error of factor + solve within 8 n eps (as a Cholesky solve's bound), and
    the same bits every time."""
    A, K, y = _problem(hs, ctx, N, bsz)
    L = hs.Cholesky(A, ctx).solve_heterogeneous().A_gpu
    b = hs.RightHandSide(N, bsz, device="cuda:0")
    runs = []
    for _ in range(3):
        b.rightHandSideData.zero_()
        b.rightHandSideData[:N] = y
        hs.TriangularSystemSolver(A, L, b, ctx).solve()
        runs.append(b.rightHandSideData.clone())
    assert torch.equal(runs[0], runs[1]) and torch.equal(runs[0], runs[2])
    x = runs[0]
    assert not x[N:].any()
    r = torch.linalg.norm(K @ x[:N] - y)
    assert r <= 8 * N * np.finfo(float).eps * torch.linalg.norm(K) * torch.linalg.norm(x)


@pytest.mark.parametrize("bsz,N", SIZES)
def test_fp32_sweeps(hs, ctx, bsz, N):
    """One application of the mixed factor: the unrefined backward error is the FP32
    factor's, well below 1e-6, and refinement with the same sweeps reaches 1e-14."""
    A, K, y = _problem(hs, ctx, N, bsz)
    b = torch.zeros(hs.padded_size(N, bsz), dtype=torch.float64, device="cuda")
    b[:N] = y
    solver = hs.MixedPrecisionSolver(A, ctx, "f16x3")
    x = solver.solve(b)
    assert solver.report["initial_backward_error"] <= 1e-6
    assert not x[N:].any()
    r = torch.linalg.norm(K @ x[:N] - y)
    assert r <= 1.1e-14 * torch.linalg.norm(K) * torch.linalg.norm(x)
