"""GPU suite: the NLML gradient where its block recurrence and its slices of blocks change
form: one block, one row past a block, few blocks and more, and each padded feature count."""
import sys
from pathlib import Path

import numpy as np
import pytest
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "oracle"))
import gp_dense as g  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bsz", [128, 256])
@pytest.mark.parametrize("N", [1, 127, 128, 129, 256, 257, 513, 1300, 2305])
@pytest.mark.parametrize("d,ard", [(1, False), (3, True), (9, True), (17, False)])
def test_gradient_at_block_edges(hs, ctx, N, bsz, d, ard):
    """cond(K) <= N sf2 / sn2 + 1 and the inverse carries some tens of eps cond(K); each
    trace is at most N / 2 beside the gradient's own size."""
    rng = np.random.default_rng(1000 * d + N)
    X = rng.random((N, d))
    y = np.sin(X.sum(1)) + 0.1 * rng.standard_normal(N)
    n_ell = d if ard else 1
    sn2 = 2e-2
    theta = np.log(np.concatenate([rng.uniform(0.5, 1.5, n_ell), [1.3, sn2]]))
    ctx.set_problem(N, bsz)
    nlml, grad, _ = hs.gp_nlml_grad(ctx, X, y, theta, n_ell=n_ell)
    nlml_ref, grad_ref = g.nlml_dense(X, y, theta, n_ell)
    tol = 64 * 2.0 ** -52 * (1.3 * N / sn2 + 1)
    assert abs(nlml - nlml_ref) <= tol * (abs(nlml_ref) + N)
    assert np.max(np.abs(grad - grad_ref)) <= tol * (np.max(np.abs(grad_ref)) + N / 2)


@pytest.mark.parametrize("N", [3072, 3073, 4865, 10100])
def test_gradient_of_many_blocks(hs, ctx, N):
    """Either side of the rule that takes the inverse to the INT8 tensor cores, and large tiles;
    the reference is the dense inverse in FP64 on the device, with the bound of the test above."""
    bsz, d, sf2, sn2 = 256, 3, 1.3, 2e-2
    g = torch.Generator(device="cuda")
    g.manual_seed(N)
    X = torch.rand((N, d), dtype=torch.float64, device="cuda", generator=g)
    y = torch.sin(X.sum(1)) + 0.1 * torch.randn(N, dtype=torch.float64, device="cuda", generator=g)
    ell = torch.tensor([0.6, 0.9, 1.4], dtype=torch.float64, device="cuda")
    theta = np.log(np.array([0.6, 0.9, 1.4, sf2, sn2]))
    ctx.set_problem(N, bsz)
    _, grad, _ = hs.gp_nlml_grad(ctx, X, y, theta)
    D = [((X[:, k, None] - X[None, :, k]) / ell[k]).square() for k in range(d)]
    Kf = sf2 * torch.exp(-0.5 * sum(D))
    L = torch.linalg.cholesky(Kf + sn2 * torch.eye(N, dtype=torch.float64, device="cuda"))
    alpha = torch.cholesky_solve(y[:, None], L)
    W = torch.cholesky_inverse(L) - alpha @ alpha.T
    ref = [0.5 * (W * Kf * Dk).sum().item() for Dk in D]
    ref += [0.5 * (W * Kf).sum().item(), 0.5 * sn2 * W.diagonal().sum().item()]
    tol = 64 * 2.0 ** -52 * (sf2 * N / sn2 + 1)
    assert np.max(np.abs(grad - ref)) <= tol * (np.max(np.abs(ref)) + N / 2)


def test_gradient_of_many_small_blocks(hs, ctx):
    """Blocks of 128 stay with the recurrence; enough of them for its large tiles."""
    N, d = 5000, 2
    rng = np.random.default_rng(N)
    X = rng.random((N, d))
    y = np.sin(X.sum(1)) + 0.1 * rng.standard_normal(N)
    theta = np.log([0.7, 1.1, 1.3, 2e-2])
    grads = []
    for bsz in (128, 256):
        ctx.set_problem(N, bsz)
        grads.append(hs.gp_nlml_grad(ctx, X, y, theta)[1])
    tol = 64 * 2.0 ** -52 * (1.3 * N / 2e-2 + 1)
    assert np.max(np.abs(grads[0] - grads[1])) <= tol * (np.max(np.abs(grads[0])) + N / 2)
