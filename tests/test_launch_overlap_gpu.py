"""Kernels that start before the one in front of them has ended: every launch that reads what the last one wrote, or writes what
it read, gives what it gives with the device idle in between, bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _lists(rs, S, lo, hi):
    return rs.randint(lo, hi + 1, S).astype(np.int64)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("S,lo,hi,H,d", [(1, 1, 1, 1, 64), (32, 4, 32, 1, 32), (24, 1, 64, 4, 64), (6, 65, 300, 2, 64), (3, 100, 700, 2, 128)])
def test_chains_without_waiting(dtype, S, lo, hi, H, d):
    from blockedattention_b200 import blockGEMM, blockSoftmax

    rs = np.random.RandomState(S + hi)
    n = _lists(rs, S, lo, hi)
    dl = np.full_like(n, d)
    g = torch.Generator("cuda").manual_seed(7)
    xs = [torch.randn((H, int(n.sum()) * d), device="cuda", generator=g).to(dtype) for _ in range(6)]

    def step(x, y, wait):
        # scores, their softmax, the product with y, which is the next step's operand
        s = blockGEMM(x, y, None, None, None, n, n, dl, scale=d ** -0.5)
        if wait:
            torch.cuda.synchronize()
        p = blockSoftmax(s, n, n)
        if wait:
            torch.cuda.synchronize()
        o = blockGEMM(p, y, None, None, None, n, dl, n, False, True)
        if wait:
            torch.cuda.synchronize()
        return s, p, o

    def run(wait):
        out, x = [], xs[0]
        for y in xs[1:]:
            r = step(x, y, wait)
            out += r
            x = r[2]
        return out

    expect = run(True)
    for _ in range(3):
        for a, b in zip(expect, run(False)):
            assert torch.equal(a, b)


def exact(q, k, v, go, n, d, scale):
    """Attention and its gradients, segment by segment in 64 bits."""
    H = q.shape[0]
    parts = []
    for x in zip(*(t.detach().cpu().double().view(H, -1, d).split(n.tolist(), 1) for t in (q, k, v, go))):
        a, b, c = (t.clone().requires_grad_(True) for t in x[:3])
        o = torch.softmax(a @ b.transpose(1, 2) * scale, -1) @ c
        parts.append((o.detach(),) + torch.autograd.grad(o, (a, b, c), x[3]))
    return [torch.cat(t, 1).reshape(H, -1) for t in zip(*parts)]


@pytest.mark.parametrize("hi,d", [(40, 64), (300, 64), (300, 128)])
def test_training_steps_without_waiting_and_captured(hi, d):
    from blockedattention_b200 import blockAttention

    rs = np.random.RandomState(hi)
    n = _lists(rs, 12, 1, hi)
    H, scale = 2, d ** -0.5
    g = torch.Generator("cuda").manual_seed(3)
    q, k, v, go = (torch.randn((H, int(n.sum()) * d), device="cuda", generator=g).half() for _ in range(4))
    for t in (q, k, v):
        t.requires_grad_(True)

    def step(wait=False):
        o = blockAttention(q, k, v, n, n, scale=scale, d=d)
        if wait:
            torch.cuda.synchronize()
        return (o.detach(),) + torch.autograd.grad(o, (q, k, v), go)

    expect = [x.clone() for x in step(True)]
    torch.cuda.synchronize()
    # (the launches of the backward pass overlap one another in that step too: it is held to 64 bits)
    for got, want in zip(expect, exact(q, k, v, go, n, d, scale)):
        got = got.cpu().double()
        assert (got - want).norm() <= 5e-3 * want.norm()
    for _ in range(4):
        for a, b in zip(expect, step()):
            assert torch.equal(a, b)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        step()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            got = step()
    for _ in range(3):
        for t in got:
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        for a, b in zip(expect, got):
            assert torch.equal(a, b)


@pytest.mark.parametrize("S,n,k,softmax", [(148, 60, 2001, False), (9, 1000, 65, True), (148, 60, 65, False)])
def test_an_early_start_costs_no_time(S, n, k, softmax):
    """Launches of one block per SM: blocks of the next kernel that settle unevenly, several on one SM, would take up to half as long
    again.  Compared with launches that a kernel of torch's, which announces nothing, keeps apart."""
    from blockedattention_b200.plan import GemmPlan

    g = torch.Generator("cuda").manual_seed(1)
    plan = GemmPlan([n] * S, [n] * S, [k] * S, 1, torch.float16, softmax=softmax, device="cuda")
    assert plan.summary["tile_items"] > 0 and plan.summary["launches"] == 1
    a, b = (torch.randn((1, d), device="cuda", generator=g).half() for d in (plan.Dm1, plan.Dm2))
    out = torch.empty((1, plan.Dout), dtype=torch.float16, device="cuda")
    small = torch.empty(1, device="cuda")

    def measure(apart):
        t = []
        for _ in range(9):
            x, y = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            torch.cuda.synchronize()
            torch.cuda._sleep(2000000)  # the launches are queued before the first one runs
            x.record()
            for _ in range(50):
                plan.run(a, b, out=out)
                if apart:
                    small.zero_()
            y.record()
            torch.cuda.synchronize()
            t.append(x.elapsed_time(y))
        return sorted(t)[4]

    measure(False)
    assert measure(False) <= 1.1 * measure(True)
