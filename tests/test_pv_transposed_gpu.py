"""GPU: the tcgen05 kernel for products with a (K, D) second operand, the first operand stored either way -- row blocks
and contraction tiles with remainders, every byte offset of a row, several items per CTA, and neighbours that hold
infinities -- against the oracle."""
import pytest
import torch

from helpers import O, assert_scores_close, packed_inputs
from blockedattention_b200.plan import GemmPlan

pytestmark = pytest.mark.gpu
M = [1, 31, 33, 64, 127, 128, 129, 257, 70, 300]
K = [1, 3, 15, 16, 17, 63, 65, 127, 128, 129, 145, 255, 256, 257, 391, 513, 777]


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("ta", [False, True])
def test_row_blocks_and_contraction_tiles(cuda_device, D, dtype, ta):
    m = [M[i % len(M)] for i in range(6 * len(K))]
    k = [K[i % len(K)] for i in range(len(m))]
    n = [D] * len(m)
    H = 4
    A, B = packed_inputs(m, n, k, H, dtype, 11, std=0.3)
    plan = GemmPlan(m, n, k, H, dtype, dtype, transpose1=ta, transpose2=True, device=cuda_device)
    assert plan.table("pv_items").size > 0
    out = torch.full((H, plan.Dout), float("nan"), dtype=dtype, device=cuda_device)
    plan.run(A.to(cuda_device), B.to(cuda_device), out=out, scale=0.5)
    plan.check()
    assert_scores_close(out, O.block_gemm(A, B, m, n, k, scale=0.5, transpose1=ta, transpose2=True), "products")
    # segments 0, 2, 4, ... hold infinities: the others must not see them
    offa = torch.tensor([0] + [x * y for x, y in zip(m, k)]).cumsum(0).tolist()
    offb = torch.tensor([0] + [x * y for x, y in zip(n, k)]).cumsum(0).tolist()
    offc = torch.tensor([0] + [x * y for x, y in zip(m, n)]).cumsum(0).tolist()
    clean = out.clone()
    for s in range(0, len(m), 2):
        A[:, offa[s]:offa[s + 1]] = float("inf")
        B[:, offb[s]:offb[s + 1]] = float("nan")
    plan.run(A.to(cuda_device), B.to(cuda_device), out=out, scale=0.5)
    plan.check()
    for s in range(1, len(m), 2):
        assert torch.equal(out[:, offc[s]:offc[s + 1]], clean[:, offc[s]:offc[s + 1]])
