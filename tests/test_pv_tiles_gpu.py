"""GPU: the P V kernel at the edges of its 256-wide tiles and 128-row value stages, with neighbours of infinities and NaN on either side
of every segment, and more items than CTAs."""
import numpy as np
import pytest
import torch

from helpers import O, assert_scores_close, packed_inputs
from blockedattention_b200.plan import GemmPlan

pytestmark = pytest.mark.gpu
K = [255, 256, 257, 383, 384, 385, 511, 512, 513, 639, 767, 769, 1, 15, 16, 17, 129, 64]
M = [1, 31, 33, 64, 97, 127, 128, 129, 200, 40]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("first", [0, 1])
def test_tiles_between_neighbours_that_are_not_finite(cuda_device, dtype, D, first):
    ks = [k for k in K for _ in range(2)] + K
    ms = [M[i % len(M)] for i in range(len(ks))]
    S, H = len(ks), 2
    ds = np.full(S, D)
    A, B = packed_inputs(ms, ds, ks, H, dtype, 3 + D)
    a1 = np.concatenate([[0], np.cumsum(np.array(ms) * np.array(ks))])
    a2 = np.concatenate([[0], np.cumsum(np.array(ks) * D)])
    ref = O.block_gemm(A, B, ms, ds, ks, transpose2=True)
    bad = torch.tensor([float("inf"), float("nan"), -float("inf")], dtype=dtype)
    for s in range(first, S, 2):  # every other segment holds nothing finite
        A[:, a1[s]:a1[s + 1]] = bad[s % 3]
        B[:, a2[s]:a2[s + 1]] = bad[(s + 1) % 3]
    plan = GemmPlan(ms, ds, ks, H, dtype, dtype, False, True, False, device=cuda_device)
    assert plan.summary["tile_items"] == 0
    out = plan.run(A.to(cuda_device), B.to(cuda_device))
    plan.check()
    ao = np.concatenate([[0], np.cumsum(np.array(ms) * D)])
    for s in range(1 - first, S, 2):
        assert_scores_close(out[:, ao[s]:ao[s + 1]], ref[:, ao[s]:ao[s + 1]], f"K={ks[s]} M={ms[s]}")


def test_more_items_than_ctas(cuda_device):
    rs = np.random.RandomState(2)
    ks, ms = rs.randint(1, 700, 300), rs.randint(1, 300, 300)
    ds = np.full(300, 128)
    A, B = packed_inputs(ms, ds, ks, 2, torch.bfloat16, 9)
    plan = GemmPlan(ms, ds, ks, 2, torch.bfloat16, torch.bfloat16, False, True, False, device=cuda_device)
    out = plan.run(A.to(cuda_device), B.to(cuda_device))
    plan.check()
    assert_scores_close(out, O.block_gemm(A, B, ms, ds, ks, transpose2=True), "P V")
