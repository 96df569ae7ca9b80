"""GPU: the backward kernels of the fused attention (16-row blocks up to 64 x 64, tcgen05 beyond) at the edges of their
tiles -- 16-row MMA steps, 32 / 64-row segments, 64-row passing tiles, 128-row resident blocks -- against torch autograd
of the per-segment formula in float64."""
import numpy as np
import pytest
import torch

from blockedattention_b200 import blockAttention, check_plans

pytestmark = pytest.mark.gpu
F16, BF16 = torch.float16, torch.bfloat16

SMALL_M = [1, 2, 15, 16, 17, 31, 32, 33, 48, 64, 64, 1]
SMALL_N = [1, 3, 16, 15, 32, 17, 31, 64, 20, 64, 1, 64]
LARGE_M = [1, 127, 128, 129, 5, 300, 0, 257, 16, 200, 65]
LARGE_N = [100, 128, 127, 129, 300, 70, 30, 65, 256, 385, 1]


def reference(q, k, v, go, m, n, d, scale):
    H = q.shape[0]
    qr, kr, vr = (t.double().requires_grad_(True) for t in (q, k, v))
    outs, oq, ok = [], 0, 0
    for ms, ns in zip(m, n):
        Q, K, V = (t[:, o * d:(o + r) * d].reshape(H, r, d) for t, o, r in ((qr, oq, ms), (kr, ok, ns), (vr, ok, ns)))
        outs.append((torch.softmax(scale * Q @ K.transpose(1, 2), -1) @ V).reshape(H, ms * d))
        oq += ms
        ok += ns
    out = torch.cat(outs, 1)
    out.backward(go.double())
    return out.detach(), qr.grad, kr.grad, vr.grad


@pytest.mark.parametrize("dtype", [F16, BF16])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("m,n,scale", [(SMALL_M, SMALL_N, 0.1), (SMALL_M, SMALL_N, -0.07), (LARGE_M, LARGE_N, 0.1),
                                       (LARGE_M, LARGE_N, -0.07), ([150, 7, 64, 700, 30], [90, 7, 65, 1500, 60], 0.1)])
def test_attention_backward_edges(cuda_device, dtype, d, m, n, scale):
    H = 3
    g = torch.Generator(device=cuda_device).manual_seed(d + len(m))

    def made(rows):
        return torch.randn((H, rows * d), generator=g, device=cuda_device).to(dtype)

    q, k, v, go = made(sum(m)), made(sum(n)), made(sum(n)), made(sum(m))
    leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
    out = blockAttention(*leaves, np.array(m), np.array(n), scale=scale, d=d)
    got = (out.detach(),) + torch.autograd.grad(out, leaves, go)
    check_plans()
    tol = 1e-2 if dtype == BF16 else 2e-3
    for name, a, b in zip(("out", "dq", "dk", "dv"), got, reference(q, k, v, go, m, n, d, scale)):
        assert torch.isfinite(a.float()).all(), name
        rel = float((a.double() - b).norm() / b.norm())
        worst = float((a.double() - b).abs().max() / b.abs().max())
        assert rel <= tol and worst <= tol, f"{name}: rel {rel}, max {worst}"


@pytest.mark.parametrize("m,n", [([20, 64], [33, 7]), ([200, 30], [70, 300])])
def test_attention_result_changed_in_place_before_backward(cuda_device, m, n):
    # a residual added to the result in place: the gradients are those of the same sum made out of place
    d, H = 64, 2
    g = torch.Generator(device=cuda_device).manual_seed(1)
    q, k, v, r = (torch.randn((H, sum(t) * d), generator=g, device=cuda_device).to(F16) for t in (m, n, n, m))
    grads = []
    for inplace in (False, True):
        leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
        out = blockAttention(*leaves, np.array(m), np.array(n), scale=0.1, d=d)
        out = out.mul_(2.0).add_(r) if inplace else out * 2.0 + r
        grads.append(torch.autograd.grad(out, leaves, r))
    assert all(torch.equal(a, b) for a, b in zip(*grads))


@pytest.mark.parametrize("dtype", [F16, BF16])
@pytest.mark.parametrize("d", [64, 128])
def test_gradient_errors_at_the_usual_scale(cuda_device, dtype, d):
    # every operand of a product is rounded to 16 bits once (P, dS and the results among them): relative roundings of half
    # a unit, 2^-12 (fp16) or 2^-9 (bf16), uniform, so 0.58 of that each in the 2-norm; an output has two or three of them
    # in a row and rowsum(dO O) one more: 2 * 2^-12 = 4.9e-4 and 2 * 2^-9 = 3.9e-3 hold all (3.1e-4 and 2.4e-3 measured)
    m, n = [300, 64, 25, 129], [300, 64, 25, 70]
    g = torch.Generator(device=cuda_device).manual_seed(d)
    q, k, v, go = (torch.randn((2, sum(t) * d), generator=g, device=cuda_device).to(dtype) for t in (m, n, n, m))
    leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
    out = blockAttention(*leaves, np.array(m), np.array(n), scale=d ** -0.5, d=d)
    got = (out.detach(),) + torch.autograd.grad(out, leaves, go)
    bound = 2 * (2.0 ** -12 if dtype == F16 else 2.0 ** -9)
    for name, a, b in zip(("out", "dq", "dk", "dv"), got, reference(q, k, v, go, m, n, d, d ** -0.5)):
        err = float((a.double() - b).norm() / b.norm())
        assert err <= bound, f"{name}: {err}"
