"""GPU suite: the fused predictive mean at the edges of its tiles (64 test x 64 training
points) and of its split over ranges of training points, against K* alpha in plain torch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 63, 64, 65, 129, 5000])
@pytest.mark.parametrize("Nt", [1, 64, 65, 700])
@pytest.mark.parametrize("d,ard", [(1, False), (8, True), (16, False), (64, True)])
def test_mean_at_tile_edges(hs, ctx, N, Nt, d, ard):
    """Each term carries a few eps (distance, exponential, product) and the sum of N terms
    N eps of the sum of their magnitudes at most: (16 d + N) eps of sum |K* alpha| (the
    d-term distance scales the exponential's argument)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(N * 1000 + Nt + d)
    X = torch.rand((N, d), dtype=torch.float64, device="cuda", generator=g)
    Xt = torch.rand((Nt, d), dtype=torch.float64, device="cuda", generator=g)
    alpha = torch.randn(N, dtype=torch.float64, device="cuda", generator=g)
    ell = torch.full((d,), 0.9, dtype=torch.float64, device="cuda")
    if ard:
        ell += 0.4 * torch.rand(d, dtype=torch.float64, device="cuda", generator=g)
    ctx.set_problem(N, 128)
    mean = hs.gp_predict(ctx, X, Xt, alpha, ell.cpu().numpy() if ard else 0.9, 1.7)
    D = torch.zeros((Nt, N), dtype=torch.float64, device="cuda")
    for k in range(d):
        D += ((Xt[:, k, None] - X[None, :, k]) / ell[k]).square()
    terms = 1.7 * torch.exp(-0.5 * D) * alpha
    bound = (16 * d + N) * 2.0 ** -52 * terms.abs().sum(dim=1)
    assert torch.all((mean - terms.sum(dim=1)).abs() <= bound)
