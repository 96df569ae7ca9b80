"""GPU: the tcgen05 GEMM kernel at the edges of its work split -- 128-column chunks, rows kept in tensor memory (512
columns) or swept twice, neighbouring items of unequal length, row blocks that fill one to four lane quarters, softmax
references that move, and the 256-column variant for long contractions -- against the oracle."""
import numpy as np
import pytest
import torch

from helpers import O, assert_probs_close, assert_scores_close, packed_inputs
from blockedattention_b200.plan import GemmPlan

pytestmark = pytest.mark.gpu
F16, BF16, F32 = torch.float16, torch.bfloat16, torch.float32
M = [1, 31, 32, 33, 64, 65, 96, 97, 128, 129, 200, 5, 70]
N = [65, 127, 128, 129, 255, 257, 383, 385, 511, 512, 513, 700, 1153]


def run(dev, M, N, K, H, dtype, out_dtype, softmax, scale, A, B):
    plan = GemmPlan(M, N, K, H, dtype, out_dtype, softmax=softmax, device=dev)
    assert plan.summary["umma_items"] > 0 and plan.summary["tile_items"] == 0
    out = torch.full((H, plan.Dout), float("nan"), dtype=out_dtype, device=dev)
    plan.run(A.to(dev), B.to(dev), out=out, scale=scale)
    plan.check()
    return plan, out


@pytest.mark.parametrize("dtype,out_dtype", [(F16, F16), (BF16, BF16), (F16, F32)])
@pytest.mark.parametrize("softmax,scale", [(True, 0.125), (True, -0.11), (False, 0.5)])
@pytest.mark.parametrize("k", [64, 72])
def test_chunks_sweeps_and_quarters(cuda_device, dtype, out_dtype, softmax, scale, k):
    m, n = M + M[::-1], N + N            # every length with two row counts
    K = [k] * len(m)
    A, B = packed_inputs(m, n, K, 3, dtype, 7)
    _, out = run(cuda_device, m, n, K, 3, dtype, out_dtype, softmax, scale, A, B)
    if softmax:
        assert_probs_close(out, O.block_scores(A, B, m, n, K, scale=scale), "softmax")
    else:
        assert_scores_close(out, O.block_gemm(A, B, m, n, K, scale=scale), "scores")


@pytest.mark.parametrize("n", [300, 500, 1400])
def test_softmax_reference_moves(cuda_device, n):
    # the second operand grows along the segment: row maxima rise by hundreds in the exponent from piece to piece
    m, n, K = [130, 40], [n, n - 37], [64, 64]
    A, B = packed_inputs(m, n, K, 2, F16, 3)
    ramp = torch.cat([torch.linspace(0.02, 6.0, x).repeat_interleave(64) for x in n])
    B = (B.float() * ramp).to(F16)
    _, out = run(cuda_device, m, n, K, 2, F16, F16, True, 1.0, A, B)
    assert_probs_close(out, O.block_scores(A, B, m, n, K, scale=1.0), "moving reference")


@pytest.mark.parametrize("out_dtype", [F16, F32])
def test_long_contractions_take_single_wide_chunks(cuda_device, out_dtype):
    m, n, K = [1, 129, 300, 70], [700, 257, 256, 515], [512, 1032, 520, 128]
    A, B = packed_inputs(m, n, K, 2, F16, 5, std=0.3)
    plan, out = run(cuda_device, m, n, K, 2, F16, out_dtype, False, 1.0, A, B)
    items = plan.table("umma_items")
    assert (items["nch"] == 1).any() and (items["nch"] == 0).any()
    assert_scores_close(out, O.block_gemm(A, B, m, n, K), "wide chunks")


@pytest.mark.parametrize("out_dtype", [F16, F32])
def test_rows_whose_offsets_exceed_32_bits(cuda_device, monkeypatch, out_dtype):
    """31 rows of such a segment are more than 2^32 elements.  Small whole numbers: every product is exact in either result type."""
    monkeypatch.setenv("BLK_UMMA_STREAMS", "0")   # (plain scores of so many tiles run on the kernel of streams otherwise)
    m, n, k = 32, 138_600_003, 16
    g = torch.Generator(device=cuda_device).manual_seed(1)
    A = torch.randint(-2, 3, (1, m * k), generator=g, device=cuda_device).half()
    B = torch.randint(-2, 3, (1, n * k), generator=g, device=cuda_device, dtype=torch.int8).half()
    plan, out = run(cuda_device, [m], [n], [k], 1, F16, out_dtype, False, 1.0, A, B)
    got, a, b = out.view(m, n), A.view(m, k), B.view(n, k)
    for c in range(0, n, 1 << 23):
        want = (a.double() @ b[c:c + (1 << 23)].double().T).to(out_dtype)
        assert torch.equal(got[:, c:c + (1 << 23)], want), f"columns from {c}"
