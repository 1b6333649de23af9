"""GPU: the reciprocal square roots of the on-chip diagonal block one by one.  For a diagonal
A_00 = diag(a) and A_10 = I the factor's first block column is L_00 = diag(sqrt(a)) and
L_10 = diag(1 / sqrt(a)), each value as the kernel forms it: two pivots a step, in a product
form within its range of sizes and one after the other outside."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


@pytest.mark.parametrize("bsz", [128, 256])
@pytest.mark.parametrize("low,high", [(-1, 1), (-100, 100), (-465, 465), (-500, 500), (462, 468), (-468, -462)])
def test_roots_and_reciprocals(hs, ctx, bsz, low, high):
    """In units of 2^-53: the iteration leaves 1.5 (half of a y's rounding, the last sum's, and a
    rest of third order), so the first of a step's two pivots has 1.5 in its reciprocal and 2.5
    in its root; the second, from the determinant's reciprocal root, 5.5 in each.  The other
    form uses sqrt and rsqrt, 1 and 2 at most."""
    rng = np.random.default_rng(bsz + abs(high))
    worst = np.zeros((2, 2))
    for _ in range(40):
        a = np.ldexp(rng.uniform(1.0, 2.0, bsz), rng.integers(low, high, bsz))
        A = hs.SymmetricMatrix(2 * bsz, bsz, device="cuda:0")
        A.block(0, 0).copy_(torch.diag(torch.from_numpy(a)))
        A.block(1, 0).copy_(torch.eye(bsz, dtype=torch.float64))
        A.block(1, 1).copy_(torch.diag(torch.from_numpy(4.0 / a)))
        hs.Cholesky(A, ctx).solve_heterogeneous()
        for i, (got, exact) in enumerate([(A.block(0, 0), np.sqrt(a.astype(np.longdouble))),
                                          (A.block(1, 0), 1 / np.sqrt(a.astype(np.longdouble)))]):
            assert torch.equal(got, torch.diag(got.diagonal()))
            v = got.diagonal().cpu().numpy()
            err = (np.abs(v - exact) / exact / U).astype(np.float64)
            worst[i] = np.maximum(worst[i], [err[0::2].max(), err[1::2].max()])
        cuda = torch.rsqrt(torch.from_numpy(a).cuda())
        d = A.block(1, 0).diagonal()
        assert ((d - cuda).abs() / cuda).max().item() <= (5.5 + 2.0) * U
    assert np.all(worst <= [[2.5, 5.5], [2.0, 5.5]]), worst
