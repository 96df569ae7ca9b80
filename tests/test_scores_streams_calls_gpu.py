"""GPU: the kernel of independent streams (blk_scores_umma.cu) as its callers reach it besides packed finite operands: token-major
operands, rows with infinities and NaN beside clean ones, and a wait that runs out."""
import numpy as np
import pytest
import torch

from helpers import O, PROB_ATOL, assert_probs_close, assert_scores_close, packed_inputs
from blockedattention_b200 import _lib as L
from blockedattention_b200.plan import GemmPlan

pytestmark = pytest.mark.gpu
F16, BF16, F32 = torch.float16, torch.bfloat16, torch.float32


@pytest.fixture(autouse=True)
def streams(monkeypatch):
    monkeypatch.setenv("BLK_UMMA_STREAMS", "1")
    monkeypatch.setenv("BLK_DISABLE_SMALL", "1")
    monkeypatch.setenv("BLK_FORCE_UMMA", "1")


@pytest.mark.parametrize("dtype,out_dtype,softmax,d", [(F16, F16, True, 64), (BF16, F32, True, 40), (BF16, BF16, False, 128), (F16, F32, False, 64)])
@pytest.mark.parametrize("H", [1, 3])
def test_token_major_operands(cuda_device, dtype, out_dtype, softmax, d, H):
    m = np.array([1, 300, 33, 128, 129, 64, 7])
    n = np.array([200, 65, 513, 1, 128, 700, 31])
    K = np.full(7, d)
    g = torch.Generator().manual_seed(d + H)
    q, k = (torch.randn((int(x.sum()), H, d), generator=g).to(dtype).to(cuda_device) for x in (m, n))
    plan = GemmPlan(m, n, K, H, dtype, out_dtype, softmax=softmax, device=cuda_device)
    assert plan.table("stream_items").size == plan.summary["umma_items"] > 0
    got = plan.run_token_major(q, k, scale=0.2)
    qs, ks = (x.permute(1, 0, 2).reshape(H, -1).contiguous() for x in (q, k))
    assert torch.equal(got, plan.run(qs, ks, scale=0.2))  # the same products, however the operands lie
    plan.check()
    if softmax:
        assert_probs_close(got, O.block_scores(qs.cpu(), ks.cpu(), m, n, K, scale=0.2), "softmax")
    else:
        assert_scores_close(got, O.block_gemm(qs.cpu(), ks.cpu(), m, n, K, scale=0.2), "scores")


@pytest.mark.parametrize("dtype,out_dtype", [(F16, F16), (BF16, BF16), (F16, F32)])
@pytest.mark.parametrize("softmax", [False, True])
@pytest.mark.parametrize("scale", [0.25, -0.25])
def test_infinities_and_nan_stay_in_their_rows(cuda_device, dtype, out_dtype, softmax, scale):
    """Segment by segment: some columns -inf; one NaN; +inf in every other row; all columns -inf; a whole tile of -inf first; clean."""
    inf, d, n = float("inf"), 64, [200, 70, 130, 300, 700, 129]
    low = -inf if scale > 0 else inf
    A, B = packed_inputs(n, n, [d] * 6, 1, dtype, 5, std=0.5)
    a = [x.view(-1, d) for x in A.split([x * d for x in n], 1)]
    b = [x.view(-1, d) for x in B.split([x * d for x in n], 1)]
    for x in a:
        x[:, 0] = 1.0
    b[0][::3, 0] = low
    b[1][5, 3] = float("nan")
    b[2][129, 0] = low
    a[2][::2, 0] = -1.0
    b[3][:, 0] = low
    b[4][:64, 0] = low
    plan = GemmPlan(n, n, [d] * 6, 1, dtype, out_dtype, softmax=softmax, device=cuda_device)
    assert plan.table("stream_items").size > 0
    out = plan.run(A.to(cuda_device), B.to(cuda_device), scale=scale)
    plan.check()
    for i, (got, x, y) in enumerate(zip(out[0].float().cpu().split([x * x for x in n]), a, b)):
        want = (x.double() @ y.double().T) * scale
        want = torch.softmax(want, -1) if softmax else want
        got = got.view(want.shape).double()
        assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf()), i
        assert torch.equal(got[want.isinf()], want[want.isinf()]), i
        fine = want.isfinite()
        # scores: half a unit of the result's type for values up to 16, and 64 products in 32 bits
        tol = PROB_ATOL if softmax else {F16: 2.0 ** -8, BF16: 2.0 ** -5, F32: 1e-4}[out_dtype]
        assert not fine.any() or (got[fine] - want[fine]).abs().max() <= tol, i
    assert torch.equal(out[0, -129 * 129:].isfinite().all().cpu(), torch.tensor(True))


@pytest.mark.parametrize("softmax", [False, True])
def test_a_wait_that_runs_out_is_reported(cuda_device, monkeypatch, softmax):
    """The producers issue no copies, so nothing is in flight when the other roles' bounded waits give up."""
    m, n, K = [300, 200, 129], [300, 600, 70], [64] * 3
    A, B = packed_inputs(m, n, K, 2, BF16, 7, std=0.5)
    plan = GemmPlan(m, n, K, 2, BF16, softmax=softmax, device=cuda_device)
    assert plan.table("stream_items").size == 3 + 2 + 2
    a, b = A.to(cuda_device), B.to(cuda_device)
    out = torch.full((2, plan.Dout), float("nan"), dtype=BF16, device=cuda_device)
    monkeypatch.setenv("BLK_TEST_STALL_PRODUCER", "1")
    plan.run(a, b, out=out, scale=0.125)
    with pytest.raises(L.BlkError) as e:
        plan.check()
    assert e.value.code == L.BLK_ERR_TIMEOUT and bool(torch.isnan(out).all())
    monkeypatch.delenv("BLK_TEST_STALL_PRODUCER")
    plan.run(a, b, out=out, scale=0.125)
    plan.check()
    if softmax:
        assert_probs_close(out, O.block_scores(A, B, m, n, K, scale=0.125), "run after a timed-out run")
    else:
        assert_scores_close(out, O.block_gemm(A, B, m, n, K, scale=0.125), "run after a timed-out run")
