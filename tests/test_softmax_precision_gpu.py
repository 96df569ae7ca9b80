"""GPU: the softmax kernel against float64 where its rounding could show -- large scores, whose exponents must not be rounded
at the scores' own size, and rows masked with a type's lowest value -- in every class of column counts."""
import numpy as np
import pytest
import torch

from blockedattention_b200 import blockSoftmax

pytestmark = pytest.mark.gpu
F16, BF16, F32 = torch.float16, torch.bfloat16, torch.float32
COLS = [1, 7, 12, 24, 60, 100, 200, 300, 500, 520, 700, 1000, 1030, 2000, 3000, 7000]  # lane, eight lanes, registers, streamed, wider than a window


def softmax(x, rows, cols, scale, device):
    flat = torch.cat([t.reshape(1, -1) for t in x], 1).to(device)
    y = blockSoftmax(flat, np.array(rows), np.array(cols), scale=scale).cpu().double()
    return [t.reshape(r, c) for t, r, c in zip(y.split([r * c for r, c in zip(rows, cols)], 1), rows, cols)]


@pytest.mark.parametrize("dtype", [F32, F16, BF16])
@pytest.mark.parametrize("size", [1.0, 30.0, 200.0, 2000.0, 20000.0])
@pytest.mark.parametrize("scale", [1.0, -0.7])
def test_error_is_relative_to_the_differences(cuda_device, dtype, size, scale):
    g = torch.Generator().manual_seed(int(size))
    rows = [37] * len(COLS)
    x = [(torch.randn((r, c), generator=g) * 2 + size).to(dtype) for r, c in zip(rows, COLS)]
    got = softmax(x, rows, COLS, scale, cuda_device)
    # the scale enters the exponent as one 32-bit factor, rounded twice (2^-23); the exponent is rounded relative to itself
    # and the exponential to 2^-22: for results above 2^-10 of their row's largest, with exponents down to -10,
    # (10 (2^-23 + 2^-24) ln 2 + 2^-22) for the element and as much again for the sum: 3e-6.  16-bit results: half a unit in
    # the last place besides
    tol = 3e-6 + {F32: 0.0, F16: 2.0 ** -11, BF16: 2.0 ** -8}[dtype]
    for a, t, c in zip(got, x, COLS):
        want = torch.softmax(t.double() * float(np.float32(scale)), -1)
        sure = (want >= want.amax(-1, keepdim=True) / 1024) & (want >= 2.0 ** -14)  # (below that a half is denormal)
        err = ((a - want).abs() / want)[sure].max().item()
        assert err <= tol, f"{c} columns: relative error {err}"


@pytest.mark.parametrize("dtype", [F32, F16, BF16])
@pytest.mark.parametrize("scale", [1.0, 0.25, -1.0, 0.0])
def test_rows_masked_with_the_lowest_value(cuda_device, dtype, scale):
    low = torch.finfo(dtype).min if scale >= 0 else torch.finfo(dtype).max
    g = torch.Generator().manual_seed(3)
    rows = [3] * len(COLS)
    x = [(torch.randn((r, c), generator=g)).to(dtype) for r, c in zip(rows, COLS)]
    for t in x:
        t[0] = low              # a row masked throughout: uniform, as torch.softmax has it
        t[1, ::2] = low         # every other column masked (all of a single column)
        t[2, 0], t[2, -1] = -low, low   # the whole range of the type in one row
    for a, t, c in zip(softmax(x, rows, COLS, scale, cuda_device), x, COLS):
        want = torch.softmax(t.double() * scale, -1)
        assert torch.isfinite(a).all(), c
        assert (a - want).abs().max().item() <= {F32: 2e-6, F16: 2.0 ** -11, BF16: 2.0 ** -8}[dtype], c
