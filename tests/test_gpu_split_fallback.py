"""GPU: where the INT8 updates' digits do not fit the device's memory, the factor and the
gradient's inverse take the FP64 tensor pipe, with the same bounds; and the mixed form's
gradient through the INT8 inverse."""
import gc

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SF2, SN2 = 1.0, 2e-2


def _data(N, d=3):
    g = torch.Generator(device="cuda")
    g.manual_seed(N)
    X = torch.rand((N, d), dtype=torch.float64, device="cuda", generator=g)
    y = torch.sin(X.sum(1)) + 0.1 * torch.randn(N, dtype=torch.float64, device="cuda", generator=g)
    return X, y


class Full:
    """The device's memory taken up but for `left` bytes."""

    def __init__(self, left):
        self.left, self.held = left, []

    def __enter__(self):
        gc.collect()
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        for _ in range(64):
            more = torch.cuda.mem_get_info()[0] - self.left
            if more < (2 << 20):
                break
            try:
                self.held.append(torch.empty(more, dtype=torch.uint8, device="cuda"))
            except torch.cuda.OutOfMemoryError:
                self.held.append(torch.empty(more // 2, dtype=torch.uint8, device="cuda"))
        return self

    def __exit__(self, *exc):
        self.held.clear()
        torch.cuda.empty_cache()


def test_gradient_without_room_for_digits(hs):
    N, theta = 3400, np.log([0.6, 0.9, 1.4, SF2, SN2])
    X, y = _data(N)
    with hs.Context(device=0, N=N, matrixBlockSize=256) as c:
        want = hs.gp_nlml_grad(c, X, y, theta)  # the INT8 inverse: 14 block rows
    with hs.Context(device=0, N=6600, matrixBlockSize=128) as c:
        # the gradient's and the solve's workspaces, and the recurrence's kernels; the digits
        # of this factor's updates are fewer than the inverse of the other takes (13 < 19 MB)
        hs.gp_nlml_grad(c, *_data(6600), theta)
        c.set_problem(1300, 256)
        hs.gp_nlml_grad(c, *_data(1300), theta)
        A, b = hs.SymmetricMatrix(N, 256, device="cuda:0"), hs.RightHandSide(N, 256, device="cuda:0")
        c.set_problem(N, 256)
        hs.MatrixGenerator.assemble(c, A.matrixData, X, 0.6, SF2, SN2)
        hs.TriangularSystemSolver(A, hs.Cholesky(A, c).solve_heterogeneous().A_gpu, b, c).solve()
        del A, b
        with Full(8 << 20):
            nlml, grad, _ = hs.gp_nlml_grad(c, X, y, theta)
    assert not np.array_equal(grad, want[1])  # it was the other path
    tol = 64 * 2.0 ** -52 * (SF2 * N / SN2 + 1)  # some tens of eps cond(K) for each
    assert abs(nlml - want[0]) <= tol * (abs(want[0]) + N)
    assert np.max(np.abs(grad - want[1])) <= tol * (np.max(np.abs(want[1])) + N / 2)


def test_factor_without_room_for_digits(hs):
    """At this size pairs of panels take 30 MB of digits, single ones 14."""
    N, bsz = 7168, 256
    X, _ = _data(N)
    A = hs.SymmetricMatrix(N, bsz, device="cuda:0")
    B = hs.SymmetricMatrix(N, bsz, device="cuda:0")
    with hs.Context(device=0, N=1300, matrixBlockSize=bsz) as c:
        small = hs.SymmetricMatrix(2000, bsz, device="cuda:0")  # loads the kernels
        hs.MatrixGenerator.assemble(c.set_problem(2000, bsz), small.matrixData, X[:2000], 0.5, SF2, SN2)
        hs.Cholesky(small, c).solve_heterogeneous()
        c.set_problem(N, bsz)
        for M in (A, B):
            hs.MatrixGenerator.assemble(c, M.matrixData, X, 0.5, SF2, SN2)
        with Full(8 << 20):
            hs.Cholesky(A, c).solve_heterogeneous()
        hs.Cholesky(B, c).solve_heterogeneous()
    assert not torch.equal(A.matrixData, B.matrixData)  # it was the other path
    nb = N // bsz
    K = torch.exp(-2.0 * torch.cdist(X, X, compute_mode="donot_use_mm_for_euclid_dist").square())
    K.diagonal().add_(SN2)
    for M in (A, B):
        L = torch.zeros((N, N), dtype=torch.float64, device="cuda")
        for j in range(nb):
            for i in range(j, nb):
                L[i * bsz:(i + 1) * bsz, j * bsz:(j + 1) * bsz] = M.block(i, j)
        # |K - L L^T| <= N u sqrt(k_ii k_jj) for a plain factor, see the INT8 update's own tests
        assert (L @ L.T - K).abs().max().item() <= 3 * N * 2.0 ** -53 * (SF2 + SN2)


@pytest.mark.parametrize("prec", ["f16x3", "tf32x3"])
def test_mixed_gradient_through_the_int8_inverse(hs, ctx, prec):
    """Blocks of 256 from 13 block rows on take the INT8 inverse, blocks of 128 the recurrence:
    both invert nearly the same low-precision factor, whose own share of the gradient is held
    to 5e-2 of its norm as for smaller sizes."""
    N, theta = 3400, np.log([0.6, 0.9, 1.4, SF2, SN2])
    X, y = _data(N)
    grads = []
    for bsz in (256, 128):
        ctx.set_problem(N, bsz)
        grads.append(hs.gp_nlml_grad(ctx, X, y, theta, precision=prec)[1])
    ctx.set_problem(N, 256)
    exact = hs.gp_nlml_grad(ctx, X, y, theta)[1]
    for got in grads:
        assert np.linalg.norm(got - exact) <= 5e-2 * np.linalg.norm(exact)


def test_solve_without_room_for_its_workspace(hs):
    """The solve's workspace (18 MB here) comes after the factor's digits (30 MB), which are given
    back for it; where even that does not help, the solve goes block by block without one."""
    N, bsz = 7168, 256
    X, y = _data(N)
    A = hs.SymmetricMatrix(N, bsz, device="cuda:0")
    b = hs.RightHandSide(N, bsz, device="cuda:0")
    K = torch.exp(-2.0 * torch.cdist(X, X, compute_mode="donot_use_mm_for_euclid_dist").square())
    K.diagonal().add_(SN2)
    with hs.Context(device=0, N=N, matrixBlockSize=bsz) as warm:
        hs.MatrixGenerator.assemble(warm, A.matrixData, X, 0.5, SF2, SN2)
        hs.TriangularSystemSolver(A, hs.Cholesky(A, warm).solve_heterogeneous().A_gpu, b, warm).solve()
        for k in (0, 1):  # loads the operators' kernels
            hs.MatrixVectorOperations.triangularSolveBlockVector(warm, A.matrixData, b.rightHandSideData, 0, 0, k)
            hs.MatrixVectorOperations.matrixVectorColumnUpdate(warm, A.matrixData, b.rightHandSideData, 1 - k, 1, k,
                                                               hs.block_id(k, k, N // bsz), N // bsz, k)
    solved = []
    for with_digits in (True, False):
        with hs.Context(device=0, N=N, matrixBlockSize=bsz) as c:
            if with_digits:
                hs.MatrixGenerator.assemble(c, A.matrixData, X, 0.5, SF2, SN2)
                hs.Cholesky(A, c).solve_heterogeneous()
            b.rightHandSideData.copy_(y)
            with Full(6 << 20):
                before = c.launch_count()
                hs.TriangularSystemSolver(A, A.matrixData, b, c).solve()
                solved.append((b.rightHandSideData.clone(), c.launch_count() - before))
    (x, few), (blockwise, many) = solved
    assert few <= 4 and many >= 2 * (N // bsz)
    for v in (x, blockwise):
        r = torch.linalg.norm(K @ v - y)
        assert r <= 8 * N * 2.0 ** -52 * torch.linalg.norm(K) * torch.linalg.norm(v)
