"""GPU: the triangular solve's workspace is the inverse diagonal blocks, a few vectors and, for
blocks of 256 only, a quadrant of scratch a block."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bsz,scratch", [(128, 0), (256, 128 * 128)])
def test_workspace_of_a_solve(hs, bsz, scratch):
    N = 12800
    nb = N // bsz
    A = hs.SymmetricMatrix(N, bsz, device="cuda:0")
    for k in range(nb):
        A.block(k, k).copy_(torch.eye(bsz, dtype=torch.float64))
    b = hs.RightHandSide(N, bsz, device="cuda:0")
    b.rightHandSideData.fill_(1.0)
    used = []
    for _ in range(2):  # the first loads the kernels
        with hs.Context(device=0, N=N, matrixBlockSize=bsz) as c:
            torch.cuda.synchronize()
            before = torch.cuda.mem_get_info()[0]
            hs.TriangularSystemSolver(A, A.matrixData, b, c).solve()
            used.append(before - torch.cuda.mem_get_info()[0])
    assert torch.all(b.rightHandSideData == 1.0)
    assert used[1] <= 8 * nb * (bsz * bsz + scratch) + 64 * N + (4 << 20)
