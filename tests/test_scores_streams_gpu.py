"""GPU: the kernel of independent streams (blk_scores_umma.cu) at the edges of its work split -- 64-column tiles, rows that begin and
end anywhere in a 32-byte sector or share one, row blocks that fill one to four lane quarters, rows swept twice, contractions of
one and two blocks -- against the oracle, with canaries around the result."""
import numpy as np
import pytest
import torch

from helpers import O, assert_probs_close, assert_scores_close, packed_inputs
from blockedattention_b200.plan import GemmPlan

pytestmark = pytest.mark.gpu
F16, BF16, F32 = torch.float16, torch.bfloat16, torch.float32
M = [1, 31, 32, 33, 64, 65, 96, 97, 128, 129, 200, 5, 70, 300, 2, 16, 127, 40]
N = [1, 5, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 191, 192, 200, 320, 511, 513]


@pytest.fixture
def streams(monkeypatch):
    monkeypatch.setenv("BLK_UMMA_STREAMS", "1")
    monkeypatch.setenv("BLK_DISABLE_SMALL", "1")
    monkeypatch.setenv("BLK_FORCE_UMMA", "1")


def run(dev, m, n, K, H, dtype, out_dtype, softmax, scale, shift):
    A, B = packed_inputs(m, n, K, H, dtype, 11)
    plan = GemmPlan(m, n, K, H, dtype, out_dtype, softmax=softmax, device=dev)
    assert plan.summary["umma_items"] > 0 and plan.summary["tile_items"] == 0
    buf = torch.full((H * plan.Dout + 64,), float("nan"), dtype=out_dtype, device=dev)
    out = buf[shift:shift + H * plan.Dout].view(H, plan.Dout)
    plan.run(A.to(dev), B.to(dev), out=out, scale=scale)
    plan.check()
    assert torch.isnan(buf[:shift]).all() and torch.isnan(buf[shift + H * plan.Dout:]).all()
    if softmax:
        assert_probs_close(out, O.block_scores(A, B, m, n, K, scale=scale), "softmax")
    else:
        assert_scores_close(out, O.block_gemm(A, B, m, n, K, scale=scale), "scores")


@pytest.mark.parametrize("dtype,out_dtype", [(F16, F16), (BF16, BF16), (F16, F32)])
@pytest.mark.parametrize("softmax,scale,k", [(True, 0.125, 64), (True, -0.11, 40), (False, 0.5, 16), (False, 1.0, 64), (False, -0.5, 72), (False, 0.3, 128)])
@pytest.mark.parametrize("shift", [0, 8])
def test_tiles_sectors_and_quarters(cuda_device, streams, dtype, out_dtype, softmax, scale, k, shift):
    n = N + N
    m = [M[i % len(M)] for i in range(len(n))]
    run(cuda_device, m, n, [k] * len(n), 3, dtype, out_dtype, softmax, scale, shift)


@pytest.mark.parametrize("softmax", [False, True])
def test_more_items_than_streams_and_mixed_contractions(cuda_device, streams, softmax):
    rs = np.random.RandomState(5)
    n = rs.randint(1, 300, 400).tolist()
    m = rs.randint(1, 200, 400).tolist()
    K = rs.choice([16, 32, 48, 64] if softmax else [16, 48, 64, 96, 128], 400).tolist()
    run(cuda_device, m, n, K, 2, F16, F32, softmax, 0.2, 0)


def test_masked_rows_and_far_scores(cuda_device, streams):
    """References that move from tile to tile, and scores beyond what one reference covers."""
    n, d, H = [700, 129], 64, 2
    K = [d, d]
    A, B = packed_inputs(n, n, K, H, BF16, 3)
    plan = GemmPlan(n, n, K, H, BF16, softmax=True, device=cuda_device)
    for scale in (3.0, -8.0):
        out = plan.run(A.to(cuda_device), B.to(cuda_device), scale=scale)
        plan.check()
        assert_probs_close(out, O.block_scores(A, B, n, n, K, scale=scale), "softmax")
    out = plan.run(A.to(cuda_device), B.to(cuda_device), scale=0.0).float()
    assert torch.allclose(out[:, :700], torch.full_like(out[:, :700], 1 / 700), rtol=8e-3)


@pytest.mark.parametrize("out_dtype,n", [(F32, 34_700_003), (F16, 69_300_003)])
def test_rows_whose_offsets_exceed_32_bits_of_bytes(cuda_device, out_dtype, n):
    """31 rows of such a segment are more than 2^32 bytes.  Small whole numbers: every product is exact in either result type."""
    m, k = 32, 16
    g = torch.Generator(device=cuda_device).manual_seed(1)
    A = torch.randint(-2, 3, (1, m * k), generator=g, device=cuda_device).half()
    B = torch.randint(-2, 3, (1, n * k), generator=g, device=cuda_device, dtype=torch.int8).half()
    plan = GemmPlan([m], [n], [k], 1, F16, out_dtype, device=cuda_device)
    out = torch.full((1, plan.Dout), float("nan"), dtype=out_dtype, device=cuda_device)
    plan.run(A, B, out=out)
    plan.check()
    got, a, b = out.view(m, n), A.view(m, k), B.view(n, k)
    for c in range(0, n, 1 << 22):
        want = (a.double() @ b[c:c + (1 << 22)].double().T).to(out_dtype)
        assert torch.equal(got[:, c:c + (1 << 22)], want), f"columns from {c}"


@pytest.mark.parametrize("out_dtype", [F16, F32])
@pytest.mark.parametrize("scale", [1.0, -1.0])
@pytest.mark.parametrize("size", [1.0, 300.0, 3000.0, 20000.0])
def test_error_is_relative_to_the_differences(cuda_device, streams, out_dtype, scale, size):
    """Probabilities of large scores that differ little.  The scores are exact: one product of `size`, the others of multiples of 1/4."""
    cols = [1, 40, 64, 65, 128, 129, 300, 512, 513, 700]
    rows, k = [37] * len(cols), [64] * len(cols)
    g = torch.Generator().manual_seed(7)
    A, B = ((torch.randint(-2, 3, (sum(x) * 64,), generator=g).float() / 4).view(-1, 64) for x in (rows, cols))
    A[:, 0], B[:, 0] = 100.0, size / 100
    A, B = A.half(), B.half()
    plan = GemmPlan(rows, cols, k, 1, F16, out_dtype, softmax=True, device=cuda_device)
    assert plan.table("stream_items").size == len(cols)
    out = plan.run(A.view(1, -1).to(cuda_device), B.view(1, -1).to(cuda_device), scale=scale).cpu().double()
    plan.check()
    # scale * log2(e) is one 32-bit factor, rounded twice (2^-23); the exponent is rounded relative to itself and the exponential
    # to 2^-22.  For results above 2^-10 of their row's largest, with exponents down to -10, (10 (2^-23 + 2^-24) ln 2 + 2^-22)
    # for the element and as much again for the sum: 3e-6.  The inverse and its product: 2^-23.  16 bits: half a unit in the last
    # place besides
    tol = 3.2e-6 + (2.0 ** -11 if out_dtype == F16 else 0.0)
    for got, a, b, n in zip(out[0].split([37 * c for c in cols]), A.double().split(rows), B.double().split(cols), cols):
        want = torch.softmax(a @ b.T * scale, -1)
        sure = (want >= want.amax(-1, keepdim=True) / 1024) & (want >= 2.0 ** -14)  # (below that a half is denormal)
        err = ((got.view(37, n) - want).abs() / want)[sure].max().item()
        assert err <= tol, f"{n} columns: relative error {err}"
