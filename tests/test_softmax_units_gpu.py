"""GPU: the pipelined softmax where its work is dealt out -- rows per warp, per eight lanes and per lane, mixed in windows
and in far more windows than the ring holds, every column class at both signs of the scale and at zero -- forward and
backward, against the oracle."""
import numpy as np
import pytest
import torch

from helpers import O, assert_probs_close
from blockedattention_b200.plan import SoftmaxPlan

pytestmark = pytest.mark.gpu
COLS = [1, 3, 8, 15, 16, 17, 31, 32, 33, 40, 63, 64, 65, 71, 200, 255, 256, 263, 264, 265, 511, 519, 520, 521, 1030, 2049, 6100]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("scale", [1.0, -0.7, 0.0])
@pytest.mark.parametrize("heads,repeat", [(1, 1), (5, 8)])
def test_units_and_ring(cuda_device, dtype, scale, heads, repeat):
    cols = np.array(COLS * repeat, np.int64)
    rows = np.array([1 + (i * 37) % 131 for i in range(len(cols))], np.int64)
    D = int((rows * cols).sum())
    g = torch.Generator().manual_seed(len(cols))
    X, G = ((torch.randn((heads, D), generator=g) * 2).to(dtype) for _ in range(2))
    plan = SoftmaxPlan(rows, cols, heads, dtype, device=cuda_device)
    out = torch.full((heads, D), float("nan"), dtype=dtype, device=cuda_device)
    plan.run(X.to(cuda_device), out=out, scale=scale)
    torch.cuda.synchronize()
    assert_probs_close(out, O.block_softmax(X, rows, cols, None, scale), "forward")
    P = out.cpu()
    grad = plan.run_backward(out, G.to(cuda_device), scale=scale).float().cpu()
    want = O.block_softmax_backward(P, G, rows, cols, scale=scale).float()
    assert (grad - want).abs().max().item() <= (1e-5 if dtype == torch.float32 else 0.02)
