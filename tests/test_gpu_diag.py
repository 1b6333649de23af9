"""GPU suite: the on-chip diagonal block (factor and inverse of one 128 or 256 block) at
the sizes and scales where it can go wrong: padding at every panel and quadrant edge,
pivots outside the range of the two-column product form, failing pivots in either column
of a step, and the inverse through the triangular solve."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _spd(N, seed, scale=1.0):
    rng = np.random.default_rng(seed)
    X = rng.random((N, 8))
    D = ((X[:, None, :] - X[None, :, :]) ** 2).sum(axis=2)
    return scale * (np.exp(-2.0 * D) + 1e-2 * np.eye(N))


def _pack(hs, K, N, bsz):
    A = hs.SymmetricMatrix(N, bsz)
    nb = A.blockCountXY
    full = np.zeros((nb * bsz, nb * bsz))
    full[:N, :N] = K
    for j in range(nb):
        for i in range(j, nb):
            A.block(i, j)[:] = torch.from_numpy(full[i * bsz:(i + 1) * bsz, j * bsz:(j + 1) * bsz].copy())
    return A


@pytest.mark.parametrize("bsz,N", [(128, n) for n in (1, 8, 31, 33, 65, 127, 128, 129, 300)] +
                         [(256, n) for n in (1, 127, 128, 129, 161, 255, 256, 257, 600)])
def test_factor_and_inverse(hs, ctx, bsz, N):
    """Backward error of the factor within n eps (the standard bound of a Cholesky factor
    is (n + 1) u ||L||_F^2-wise, u = eps / 2), the solution's within 8 n eps."""
    eps = np.finfo(float).eps
    K = _spd(N, N + bsz)
    A = _pack(hs, K, N, bsz)
    chol = hs.Cholesky(A, ctx).solve_heterogeneous()
    L = np.tril(A.to_dense())
    for k in range(A.blockCountXY):
        assert not np.triu(A.block(k, k).numpy(), 1).any()
    assert np.linalg.norm(L @ L.T - K) <= N * eps * np.linalg.norm(K)
    b = hs.RightHandSide(N, bsz)
    y = np.sin(np.arange(N))
    b.rightHandSideData[:N] = torch.from_numpy(y)
    hs.TriangularSystemSolver(A, chol.A_gpu, b, ctx).solve()
    x = b.rightHandSideData.numpy()
    assert not x[N:].any()
    assert np.linalg.norm(K @ x[:N] - y) <= 8 * N * eps * np.linalg.norm(K) * np.linalg.norm(x)


@pytest.mark.parametrize("bsz", [128, 256])
@pytest.mark.parametrize("scale", [2.0 ** -700, 2.0 ** -480, 2.0 ** 480, 2.0 ** 700])
def test_scales_outside_the_product_form(hs, ctx, bsz, scale):
    """A power-of-four scale is exact in L: the factor stays within n eps of sqrt(scale)
    times the unscaled matrix's (the general path against the product form)."""
    N = bsz + 40
    K = _spd(N, 3)
    A, B = _pack(hs, K, N, bsz), _pack(hs, K * scale, N, bsz)
    hs.Cholesky(A, ctx).solve_heterogeneous()
    hs.Cholesky(B, ctx).solve_heterogeneous()
    L, M = np.tril(A.to_dense()), np.tril(B.to_dense()) / np.sqrt(scale)
    assert np.linalg.norm(M @ M.T - K) <= N * np.finfo(float).eps * np.linalg.norm(K)
    assert np.linalg.norm(L - M) <= 1e-12 * np.linalg.norm(L)


@pytest.mark.parametrize("bsz", [128, 256])
@pytest.mark.parametrize("row", [0, 1, 30, 63, 64, 127, 128, 201])
@pytest.mark.parametrize("value", [-1.0, 0.0, float("nan")])
def test_failing_pivot_is_reported(hs, ctx, bsz, row, value):
    N = 210
    K = np.eye(N)
    K[row, row] = value
    A = _pack(hs, K, N, bsz)
    chol = hs.Cholesky(A, ctx)
    with pytest.raises(hs.NotSPDError):
        chol.solve_heterogeneous()
    assert chol.info == row
