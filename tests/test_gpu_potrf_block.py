"""GPU: the factor of one diagonal block as a call of its own: no scratch (so it can be captured
before any other call), any alignment of doubles, padding rows untouched but for their diagonal."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _block(N, bsz, offset=0):
    """An SPD N x N corner in a bsz x bsz block of noise, `offset` doubles into its storage."""
    rng = np.random.default_rng(N + bsz)
    M = rng.uniform(1.0, 2.0, (bsz, bsz))
    B = rng.standard_normal((N, N))
    K = B @ B.T / N + np.eye(N)
    M[:N, :N] = K
    store = torch.zeros(offset + bsz * bsz, dtype=torch.float64, device="cuda")
    A = store[offset:]
    A.copy_(torch.from_numpy(M.reshape(-1)))
    return A, M, K


def _check(A, M, K, N, bsz):
    """Backward error within N eps; the zeros above the diagonal of valid rows; padding rows."""
    out = A.cpu().numpy().reshape(bsz, bsz)
    L = np.tril(out[:N, :N])
    assert np.linalg.norm(L @ L.T - K) <= N * np.finfo(float).eps * np.linalg.norm(K)
    assert not np.triu(out[:N], 1).any()
    pad = M[N:].copy()
    i = np.arange(bsz - N)
    pad[i, N + i] = np.sqrt(pad[i, N + i])
    assert np.array_equal(out[N:], pad)


@pytest.mark.parametrize("bsz,N", [(128, n) for n in (1, 33, 127, 128)] + [(256, n) for n in (1, 127, 128, 129, 200, 256)])
@pytest.mark.parametrize("offset", [0, 1])
def test_in_place_factor(hs, ctx, bsz, N, offset):
    ctx.set_problem(N, bsz)
    A, M, K = _block(N, bsz, offset)
    hs.MatrixOperations.cholesky(ctx, A, 0, 0)
    assert ctx.take_info() == -1
    _check(A, M, K, N, bsz)


@pytest.mark.parametrize("bsz,N", [(128, 100), (128, 128), (256, 100)])
def test_factor_of_one_block_at_any_alignment(hs, ctx, bsz, N):
    A = hs.SymmetricMatrix(N, bsz, device="cuda:0")
    A.matrixData, M, K = _block(N, bsz, 1)
    hs.Cholesky(A, ctx).solve_heterogeneous()
    _check(A.matrixData, M, K, N, bsz)


def test_several_blocks_want_16_bytes(hs, ctx):
    """Refused on the host (the copies into shared memory always needed it)."""
    A = hs.SymmetricMatrix(300, 128, device="cuda:0")
    A.matrixData = torch.zeros(A.matrixData.numel() + 1, dtype=torch.float64, device="cuda")[1:]
    b = hs.RightHandSide(300, 128, device="cuda:0")
    for call in (hs.Cholesky(A, ctx).solve_heterogeneous, hs.TriangularSystemSolver(A, A.matrixData, b, ctx).solve,
                 hs.CG(A, b, ctx).solveHeterogeneous):
        with pytest.raises(hs.HSError, match="16 bytes"):
            call()


@pytest.mark.parametrize("bsz,N", [(128, 128), (256, 256)])
def test_capture_as_the_first_call(hs, bsz, N):
    stream = torch.cuda.Stream()
    A, M, K = _block(N, bsz)
    torch.cuda.synchronize()
    with hs.Context(device=0, stream=stream, N=N, matrixBlockSize=bsz) as c:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            hs.MatrixOperations.cholesky(c, A, 0, 0)
        A.copy_(torch.from_numpy(M.reshape(-1)))
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert c.take_info() == -1
        _check(A, M, K, N, bsz)
