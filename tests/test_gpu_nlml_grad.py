"""GPU suite: the NLML gradient where its block recurrence and its slices of blocks change
form: one block, one row past a block, few blocks and more, and each padded feature count."""
import sys
from pathlib import Path

import numpy as np
import pytest

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
