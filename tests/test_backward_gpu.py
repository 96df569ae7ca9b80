"""GPU: the backward pair -- softmax backward kernel and the two permuted GEMM launches -- against the oracle,
and the autograd surface of the Python operators (upstream test/pytest.py:43-46 runs ``res.mean().backward()``)."""
import numpy as np
import pytest
import torch

from helpers import O, packed_inputs
from blockedattention_b200 import blockAttention, blockAttnScores, blockGEMM, blockSoftmax
from blockedattention_b200.plan import SoftmaxPlan

pytestmark = pytest.mark.gpu
F16, BF16, F32 = torch.float16, torch.bfloat16, torch.float32
TOL = {F32: 2e-5, F16: 2e-3, BF16: 1.6e-2}


def close(got, want, dtype, what):
    got = got.detach().float().cpu(); want = want.float()
    scale = max(1.0, float(want.abs().max()))
    err = float((got - want).abs().max())
    assert err <= TOL[dtype] * scale, f"{what}: max abs err {err} (scale {scale})"


@pytest.mark.parametrize("dtype", [F32, F16, BF16])
def test_softmax_backward_kernel(cuda_device, dtype):
    dev = cuda_device
    rs = np.random.RandomState(11)
    # short rows (sub-warp groups), rows of a few hundred columns, a row longer than the 16 KB window, odd offsets
    rows = np.array([5, 1, 17, 3, 2, 40, 1, 7]); cols = np.array([3, 1, 33, 700, 9000, 64, 5000, 129])
    H = 3
    D = int((rows * cols).sum())
    X = torch.randn(H, D) * 2
    P = O.block_softmax(X, rows, cols, scale=0.9).to(dtype)
    G = torch.randn(H, D).to(dtype)
    plan = SoftmaxPlan(rows, cols, H, dtype, device=dev)
    got = plan.run_backward(P.to(dev), G.to(dev), scale=0.9)
    want = O.block_softmax_backward(P, G, rows, cols, scale=0.9)
    close(got, want, dtype, "softmax backward")
    # in place on the gradient
    g2 = G.to(dev).clone()
    res = plan.run_backward(P.to(dev), g2, grad_src=g2, scale=0.9)
    assert res.data_ptr() == g2.data_ptr() and torch.equal(res, got)
    # offsets with gaps: untouched elements keep their canary
    acc = np.concatenate([[0], np.cumsum(rows * cols + 3)])
    Dg = int(acc[-1])
    Pg = torch.zeros(H, Dg, dtype=dtype); Gg = torch.zeros(H, Dg, dtype=dtype)
    for s in range(len(rows)):
        n = int(rows[s] * cols[s]); o = int((rows[:s] * cols[:s]).sum())
        Pg[:, acc[s]:acc[s] + n] = P[:, o:o + n]; Gg[:, acc[s]:acc[s] + n] = G[:, o:o + n]
    plan_g = SoftmaxPlan(rows, cols, H, dtype, accum=acc, device=dev)
    out = torch.full((H, Dg), 7.0, dtype=dtype, device=dev)
    plan_g.run_backward(Pg.to(dev), Gg.to(dev), grad_src=out, scale=0.9)
    want_g = O.block_softmax_backward(Pg, Gg, rows, cols, srcAccum=acc, scale=0.9)
    for s in range(len(rows)):
        n = int(rows[s] * cols[s])
        close(out[:, acc[s]:acc[s] + n], want_g[:, acc[s]:acc[s] + n], dtype, f"gapped segment {s}")
        assert bool((out[:, acc[s] + n:acc[s + 1]] == 7.0).all())


@pytest.mark.parametrize("dtype,K", [(F32, 24), (F16, 64), (BF16, 40)])
def test_gemm_autograd_matches_upstream_backward(cuda_device, dtype, K):
    dev = cuda_device
    rs = np.random.RandomState(7)
    M = rs.randint(1, 90, size=12); N = rs.randint(1, 90, size=12); Kl = np.full(12, K)
    H = 2
    A, B = packed_inputs(M, N, Kl, H, dtype, 4)
    a = A.to(dev).requires_grad_(); b = B.to(dev).requires_grad_()
    out = blockGEMM(a, b, None, None, None, M, N, Kl, scale=0.5)
    assert out.requires_grad
    g = (torch.randn(out.shape) * 0.5).to(dtype)
    out.backward(g.to(dev))
    w1, w2 = O.block_gemm_backward(A, B, g, M, N, Kl, scale=0.5)
    close(a.grad, w1, dtype, "mat1 grad")
    close(b.grad, w2, dtype, "mat2 grad")
    assert a.grad.shape == a.shape and b.grad.shape == b.shape and a.grad.dtype == dtype


def test_chained_operators_backward_like_upstream_script(cuda_device):
    # blockGEMM -> blockSoftmax -> mean().backward(), fp32, the upstream script's sizes (test/pytest.py:7-46)
    dev = cuda_device
    h, m, n, k = 8, 33, 99, 64
    M = torch.tensor([m, n, k], device=dev); Kl = torch.tensor([k, k, k], device=dev)
    torch.manual_seed(0)
    A = torch.randn(h, m * k + n * k + k * k); B = torch.randn(h, m * k + n * k + k * k)
    a = A.to(dev).requires_grad_(); b = B.to(dev).requires_grad_()
    res = blockSoftmax(blockGEMM(a, b, None, None, None, M, M, Kl), M, M)
    res.mean().backward()
    # the same chain with torch autograd on the CPU, float64
    a64 = A.double().requires_grad_(); b64 = B.double().requires_grad_()
    outs, o = [], 0
    for r in (m, n, k):
        x = a64[:, o:o + r * k].reshape(h, r, k); y = b64[:, o:o + r * k].reshape(h, r, k)
        outs.append((x @ y.transpose(1, 2)).softmax(-1).reshape(h, r * r)); o += r * k
    torch.cat(outs, 1).mean().backward()
    close(a.grad, a64.grad, F32, "chained mat1 grad")
    close(b.grad, b64.grad, F32, "chained mat2 grad")


@pytest.mark.parametrize("dtype", [F16, BF16])
def test_fused_scores_backward(cuda_device, dtype):
    dev = cuda_device
    rs = np.random.RandomState(2)
    n = rs.randint(2, 70, size=20); Kl = np.full(20, 64)
    H = 4
    Q, Kt = packed_inputs(n, n, Kl, H, dtype, 9)
    q = Q.to(dev).requires_grad_(); k = Kt.to(dev).requires_grad_()
    p = blockAttnScores(q, k, n, n, Kl, scale=0.125)
    g = torch.randn(p.shape).to(dtype)
    p.backward(g.to(dev))
    # oracle: softmax backward on the rounded probabilities, then the two permuted GEMMs with the scale
    ds = O.block_softmax_backward(p.detach().cpu(), g, n, n).to(dtype)
    w1, w2 = O.block_gemm_backward(Q, Kt, ds, n, n, Kl, scale=0.125)
    close(q.grad, w1, dtype, "dq")
    close(k.grad, w2, dtype, "dk")


@pytest.mark.parametrize("d,sizes", [(64, [5, 33, 64, 17]),          # packs of the small-segment kernel
                                     (64, [5, 200, 64, 130]),        # packs and the tcgen05 attention kernel
                                     (128, [150, 7, 260])])          # the tcgen05 attention kernel
def test_fused_attention_backward(cuda_device, d, sizes):
    # forward on the fused kernels, backward on kernels of its own that recompute the probabilities.  Checked against
    # torch autograd of the per-segment formula in float64.
    dev = cuda_device
    n = np.array(sizes, np.int64)
    m = np.maximum(n - 3, 1)                      # fewer queries than keys
    H, scale = 2, 0.1
    g = torch.Generator().manual_seed(5)
    q0 = torch.randn((H, int(m.sum()) * d), generator=g).to(F16)
    k0 = torch.randn((H, int(n.sum()) * d), generator=g).to(F16)
    v0 = torch.randn((H, int(n.sum()) * d), generator=g).to(F16)
    go = torch.randn((H, int(m.sum()) * d), generator=g).to(F16)
    q, k, v = (t.to(dev).requires_grad_(True) for t in (q0, k0, v0))
    out = blockAttention(q, k, v, m, n, scale=scale, d=d)
    out.backward(go.to(dev))
    # reference
    qr, kr, vr = (t.double().requires_grad_(True) for t in (q0, k0, v0))
    outs = []; oq = okv = 0
    for ms, ns in zip(m, n):
        ms, ns = int(ms), int(ns)
        Q = qr[:, oq * d:(oq + ms) * d].reshape(H, ms, d); K = kr[:, okv * d:(okv + ns) * d].reshape(H, ns, d)
        V = vr[:, okv * d:(okv + ns) * d].reshape(H, ns, d)
        outs.append((torch.softmax(scale * Q @ K.transpose(1, 2), dim=-1) @ V).reshape(H, ms * d))
        oq += ms; okv += ns
    ref = torch.cat(outs, dim=1)
    ref.backward(go.double())
    close(out, ref.detach(), F16, "fused attention forward")
    for name, got, want in (("dq", q.grad, qr.grad), ("dk", k.grad, kr.grad), ("dv", v.grad, vr.grad)):
        assert got is not None and got.shape == want.shape
        s = max(1.0, float(want.abs().max()))
        err = float((got.float().cpu() - want.float()).abs().max())
        assert err <= 1e-2 * s, f"{name}: max abs err {err} (scale {s})"


def test_library_errors_of_a_backward_pass_keep_their_class(cuda_device, monkeypatch):
    # the gradient's own launch gives up a bounded wait (see test_timeout_gpu.py): the caller of backward() must get the
    # same BlkError with its code as the caller of an operator
    from blockedattention_b200 import _lib as L
    dev, n = cuda_device, np.array([200, 136])
    k = np.array([64, 64])
    a = torch.randn((1, int((n * k).sum())), device=dev).half().requires_grad_()
    b = torch.randn((1, int((n * k).sum())), device=dev).half()          # stored (k, n): the gradient of a is a plain product
    out = blockGEMM(a, b, None, None, None, n, n, k, False, True)
    g = torch.randn_like(out)
    monkeypatch.setenv("BLK_CHECK", "1")
    monkeypatch.setenv("BLK_TEST_STALL_PRODUCER", "1")
    with pytest.raises(L.BlkError) as e:
        out.backward(g, retain_graph=True)
    assert e.value.code == L.BLK_ERR_TIMEOUT
    monkeypatch.delenv("BLK_TEST_STALL_PRODUCER")
    out.backward(g)
    want = O.block_gemm_backward(a.detach().cpu(), b.cpu(), g.cpu(), n, n, k, transpose2=True)[0]
    close(a.grad, want, F16, "mat1 grad after a failed pass")


def _attention(q, k, v, n, d):
    return blockAttention(q, k, v, n, n, scale=0.1, d=d)


@pytest.mark.parametrize("op", ["gemm", "scores", "softmax", "attention"])
def test_saved_tensor_hooks(cuda_device, op):
    # what a hook hands back is checked before a kernel reads it: another type is converted, a tensor on the host, of
    # another size or not contiguous is refused (all of these on purpose do not reach a launch)
    dev, d, n = cuda_device, 64, np.array([40, 100])
    D, kl = int((n * 64).sum()), np.array([64, 64])
    S = int((n * n).sum())
    call, sizes = {"gemm": (lambda a, b: blockGEMM(a, b, None, None, None, n, n, kl), (D, D)),
                   "scores": (lambda a, b: blockAttnScores(a, b, n, n, kl), (D, D)),
                   "softmax": (lambda a: blockSoftmax(a, n, n), (S,)),
                   "attention": (lambda a, b, c: _attention(a, b, c, n, d), (D, D, D))}[op]
    g = torch.Generator(device=dev).manual_seed(4)
    base = [(torch.randn((2, s), generator=g, device=dev) * 0.3).half() for s in sizes]
    go = None

    def grads(pack, unpack):
        nonlocal go
        leaves = [t.clone().requires_grad_(True) for t in base]
        with torch.autograd.graph.saved_tensors_hooks(pack, unpack):
            out = call(*leaves)
        if go is None:
            go = (torch.randn(out.shape, generator=g, device=dev)).half()
        return torch.autograd.grad(out, leaves, go)

    same = lambda x: x
    want = grads(same, same)
    for pack, unpack in ((lambda x: x.cpu(), lambda x: x.to(dev)), (same, lambda x: x.double().to(x.dtype)),
                         (same, lambda x: x.float() if x.dtype == F16 else x)):
        assert all(torch.equal(a, b) for a, b in zip(grads(pack, unpack), want))
    for unpack in (lambda x: x.cpu(), lambda x: x[:, :-8], lambda x: x[:1], lambda x: torch.cat([x, x], 1)[:, ::2],
                   lambda x: torch.stack([x, x], -1)[..., 0]):
        with pytest.raises(RuntimeError):
            grads(same, unpack)
    assert all(torch.equal(a, b) for a, b in zip(grads(same, same), want))


@pytest.mark.parametrize("op", ["gemm", "scores", "softmax", "attention"])
def test_forward_mode_is_refused_not_dropped(cuda_device, op):
    import torch.autograd.forward_ad as fwAD
    dev, n, kl = cuda_device, np.array([20, 70]), np.array([64, 64])
    x, s = (torch.randn((2, int((n * t).sum())), device=dev).half() for t in (kl, n))
    with fwAD.dual_level():
        dual = lambda t: fwAD.make_dual(t.clone().requires_grad_(True), torch.ones_like(t))
        with pytest.raises(NotImplementedError):
            if op == "softmax":
                blockSoftmax(dual(s), n, n)
            elif op == "attention":
                blockAttention(x, dual(x), x, n, n, d=64)
            else:
                (blockGEMM if op == "gemm" else blockAttnScores)(*((x, dual(x)) + ((None,) * 3 if op == "gemm" else ())), n, n, kl)
