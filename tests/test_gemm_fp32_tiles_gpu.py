"""GPU: the fp32 GEMM at the edges of its 128 x 128 and 64 x 64 tiles and its steps of 16, rows of any alignment, either operand
transposed.  The operands are small integers, whose products and sums fp32 holds exactly: results are equal, not close."""
import numpy as np
import pytest
import torch

from helpers import O
from blockedattention_b200.plan import GemmPlan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ta,tb", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("H,mult", [(30, 1), (2, 1), (30, 4)])
def test_tiles_of_both_sizes(cuda_device, ta, tb, H, mult):
    rs = np.random.RandomState(H + mult)
    M = [128, 127, 129, 1, 64, 65, 256, 257, 200, 100, 5, 132, 260, 96]
    N = [128, 129, 127, 200, 65, 64, 100, 256, 3, 300, 7, 124, 128, 60]
    K = [1, 3, 4, 15, 16, 17, 31, 32, 33, 64, 70, 100, 20, 48]
    if mult > 1:  # rows of whole vectors
        M, N, K = ([-(-x // mult) * mult for x in y] for y in (M, N, K))
    D1, D2 = int(np.dot(M, K)), int(np.dot(N, K))
    A = torch.from_numpy(rs.randint(-4, 5, (H, D1)).astype(np.float32))
    B = torch.from_numpy(rs.randint(-4, 5, (H, D2)).astype(np.float32))
    plan = GemmPlan(M, N, K, H, torch.float32, torch.float32, ta, tb, False, device=cuda_device)
    assert plan.summary["launches"] == (2 if H > 2 else 1)
    buf = torch.full((H * plan.Dout + 16,), float("nan"), device=cuda_device)
    plan.run(A.to(cuda_device), B.to(cuda_device), out=buf[4:4 + H * plan.Dout].view(H, -1), scale=0.5)
    plan.check()
    assert torch.isnan(buf[:4]).all() and torch.isnan(buf[4 + H * plan.Dout:]).all()
    ref = O.block_gemm(A, B, M, N, K, transpose1=ta, transpose2=tb, scale=0.5)
    assert torch.equal(buf[4:4 + H * plan.Dout].view(H, -1).cpu(), ref)
