"""GPU: a prediction's partial sums fit the scratch that every context has after its first call, so
no later call of any size allocates; a capture, in which nothing may, shows it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,Nt", [(16384, 5000), (16384, 6000), (3000, 100), (20000, 56000), (30000, 1000), (700, 70000)])
def test_no_growth_after_the_first_call(hs, N, Nt):
    stream = torch.cuda.Stream()
    d = 4
    with torch.cuda.stream(stream), hs.Context(device=0, stream=stream, N=N, matrixBlockSize=128) as c:
        g = torch.Generator(device="cuda")
        g.manual_seed(N + Nt)
        X = torch.rand((N, d), dtype=torch.float64, device="cuda", generator=g)
        Xt = torch.rand((Nt, d), dtype=torch.float64, device="cuda", generator=g)
        alpha = torch.randn(N, dtype=torch.float64, device="cuda", generator=g)
        hs.gp_predict(c, X, Xt[:1], alpha, 0.5, 1.0)
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            mean = hs.gp_predict(c, X, Xt, alpha, 0.5, 1.0)
        graph.replay()
        assert torch.equal(mean, hs.gp_predict(c, X, Xt, alpha, 0.5, 1.0))
        # sums of N terms of size |alpha| in another order
        j = torch.arange(0, Nt, max(1, Nt // 50), device="cuda")
        K = torch.exp(-2.0 * torch.cdist(Xt[j], X, compute_mode="donot_use_mm_for_euclid_dist").square())
        assert (mean[j] - K @ alpha).abs().max() <= 2 * N * 2.0 ** -53 * alpha.abs().sum()
