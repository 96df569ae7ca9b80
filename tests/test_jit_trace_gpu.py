"""GPU: torch.jit.trace over the operators -- a replay computes on the replay's inputs, with and without gradients."""
import numpy as np
import pytest
import torch

from blockedattention_b200 import (blockAttention, blockAttentionTokenMajor, blockAttnScores, blockAttnScoresTokenMajor,
                                   blockGEMM, blockSoftmax)

pytestmark = pytest.mark.gpu
N, KL, D = np.array([20, 70]), np.array([64, 64]), 64
ROWS, CELLS = int(N.sum()), int((N * N).sum())
TOKENS = (ROWS, 2, D)
OPS = {"gemm": (lambda a, b: blockGEMM(a, b, None, None, None, N, N, KL, scale=0.5), [(2, ROWS * D)] * 2),
       "gemm, fp32 result": (lambda a, b: blockGEMM(a, b, None, None, None, N, N, KL, out_dtype=torch.float32), [(2, ROWS * D)] * 2),
       "scores": (lambda a, b: blockAttnScores(a, b, N, N, KL, scale=0.1), [(2, ROWS * D)] * 2),
       "softmax": (lambda a: blockSoftmax(a, N, N), [(2, CELLS)]),
       "chain": (lambda a, b: blockSoftmax(blockGEMM(a, b, None, None, None, N, N, KL, scale=0.1) * 1.0, N, N), [(2, ROWS * D)] * 2),
       "attention": (lambda a, b, c: blockAttention(a, b, c, N, N, scale=0.1, d=D), [(2, ROWS * D)] * 3),
       "attention, tokens": (lambda a, b, c: blockAttentionTokenMajor(a, b, c, N, scale=0.1), [TOKENS] * 3),
       "scores, tokens": (lambda a, b: blockAttnScoresTokenMajor(a, b, N, scale=0.1), [TOKENS] * 2)}


@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("name", OPS)
def test_trace_and_replay(cuda_device, name, grad):
    call, shapes = OPS[name]
    grad = grad and "tokens" not in name     # forward only
    g = torch.Generator(device=cuda_device).manual_seed(1)
    made = lambda: [torch.randn(s, generator=g, device=cuda_device).half().requires_grad_(grad) for s in shapes]
    traced = torch.jit.trace(call, tuple(made()), check_trace=False)
    for _ in range(2):
        ins = made()
        want, got = call(*ins), traced(*ins)
        assert torch.equal(got, want)
        if grad:
            go = torch.randn(want.shape, generator=g, device=cuda_device).to(want.dtype)
            assert all(torch.equal(a, b) for a, b in zip(torch.autograd.grad(got, ins, go), torch.autograd.grad(want, ins, go)))
