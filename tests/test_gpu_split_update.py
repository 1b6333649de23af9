"""GPU suite: the FP64 factor where its trailing update runs on the INT8 tensor cores: either
side of the rule, ragged last blocks, rows of very different sizes, and rows whose digits
take the ends of their range."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _blocks(hs, N, bsz):
    nb = -(-N // bsz)
    for j in range(nb):
        for i in range(j, nb):
            yield i * bsz, j * bsz, hs.block_id(i, j, nb) * bsz * bsz


def _pack(hs, K, N, bsz):
    n = -(-N // bsz) * bsz
    full = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    full[:N, :N] = K.tril()
    out = torch.zeros(hs.packed_size(N, bsz), dtype=torch.float64, device="cuda")
    for r, c, s in _blocks(hs, N, bsz):
        out[s:s + bsz * bsz] = full[r:r + bsz, c:c + bsz].reshape(-1)
    return out


def _factor(hs, ctx, K, N, bsz):
    A = hs.SymmetricMatrix(N, bsz, device="cuda:0")
    A.matrixData.copy_(_pack(hs, K, N, bsz))
    packed = hs.Cholesky(A, ctx).solve_heterogeneous().A_gpu
    n = -(-N // bsz) * bsz
    L = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    for r, c, s in _blocks(hs, N, bsz):
        L[r:r + bsz, c:c + bsz] = packed[s:s + bsz * bsz].view(bsz, bsz)
    return L


def _matrix(kind, N):
    g = torch.Generator(device="cuda")
    g.manual_seed(N)
    X = torch.rand((N, 8), dtype=torch.float64, device="cuda", generator=g)
    if kind == "wishart":
        B = torch.randn((N, N), dtype=torch.float64, device="cuda", generator=g)
        return B @ B.T / N + 0.1 * torch.eye(N, dtype=torch.float64, device="cuda")
    if kind == "constant":  # factor columns of equal entries
        return torch.full((N, N), 0.99, dtype=torch.float64, device="cuda") + 0.01 * torch.eye(N, dtype=torch.float64, device="cuda")
    d2 = torch.cdist(X, X, compute_mode="donot_use_mm_for_euclid_dist") ** 2
    K = torch.exp(-0.5 * d2 / 0.36) + 1e-2 * torch.eye(N, dtype=torch.float64, device="cuda")
    if kind == "scaled":
        s = 10.0 ** (120 * torch.rand(N, dtype=torch.float64, device="cuda", generator=g) - 60)
        K = K * s[:, None] * s[None, :]
    return K


@pytest.mark.parametrize("kind", ["rbf", "scaled", "wishart", "constant"])
@pytest.mark.parametrize("N,bsz", [(2300, 256), (2560, 256), (2561, 256), (7168, 256), (7425, 256), (3400, 128), (3584, 128), (6657, 128)])
def test_backward_error(hs, ctx, kind, N, bsz):
    """|A - L L^T|_ij <= N u sqrt(a_ii a_jj) for a plain factor, twice that where products of
    256 terms carry 2^-57 of their scales each, and N u for the product formed here."""
    K = _matrix(kind, N)
    ctx.set_problem(N, bsz)
    L = _factor(hs, ctx, K, N, bsz)
    assert torch.all(L[N:, :] == 0.0) and torch.all(L.triu(1)[:N] == 0.0)
    L = L[:N, :N]
    s = K.diagonal().sqrt()
    # the rows' scales taken out first: their products could leave the range
    Ls = L / s[:, None]
    err = (Ls @ Ls.T - K / s[:, None] / s[None, :]).abs().max().item()
    assert err <= 3 * N * 2.0 ** -53


@pytest.mark.parametrize("bad", [-1.0, float("nan")])
@pytest.mark.parametrize("row", [40, 1500, 2999])
def test_failing_pivot_is_named(hs, ctx, bad, row):
    N, bsz = 3000, 256
    K = _matrix("wishart", N)
    K[row, row] = bad
    ctx.set_problem(N, bsz)
    with pytest.raises(Exception, match=f"row {row}"):
        _factor(hs, ctx, K, N, bsz)
