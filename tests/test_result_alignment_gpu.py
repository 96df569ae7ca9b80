"""GPU: results that lie on 32-byte sectors leave the tcgen05 kernels as sectors, others as 16-byte vectors: the same numbers, and
nothing around them touched."""
import numpy as np
import pytest
import torch

from helpers import packed_inputs
from blockedattention_b200.plan import AttentionPlan, GemmPlan

pytestmark = pytest.mark.gpu


def both(numel, dtype, dev, run):
    got = []
    for shift in (0, 8, 16):
        buf = torch.full((numel + 32,), float("nan"), dtype=dtype, device=dev)
        run(buf[shift:shift + numel])
        assert torch.isnan(buf[:shift]).all() and torch.isnan(buf[shift + numel:]).all()
        got.append(buf[shift:shift + numel].clone())
    assert not torch.isnan(got[0]).any()
    for x in got[1:]:
        assert torch.equal(x, got[0])


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("d", [64, 128])
def test_results_on_and_off_sectors(cuda_device, dtype, d):
    n = np.array([1, 31, 65, 128, 129, 200, 300, 97])
    H = 3
    q, k = (x.to(cuda_device) for x in packed_inputs(n, n, np.full_like(n, d), H, dtype, d))
    v = packed_inputs(n, n, np.full_like(n, d), H, dtype, d + 1)[0].to(cuda_device)
    plan = AttentionPlan(n, n, H, dtype, device=cuda_device, d=d)
    numel = H * int(n.sum()) * d
    both(numel, dtype, cuda_device, lambda out: plan.run(q, k, v, out=out.view(H, -1), scale=0.1))
    plan.check()
    probs = GemmPlan(n, n, np.full_like(n, d), H, dtype, softmax=True, device=cuda_device).run(q, k, scale=0.1)
    pv = GemmPlan(n, np.full_like(n, d), n, H, dtype, dtype, False, True, False, device=cuda_device)
    both(numel, dtype, cuda_device, lambda out: pv.run(probs, v, out=out.view(H, -1)))
    pv.check()
