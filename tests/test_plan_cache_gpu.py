"""GPU: what the operators remember -- plans under the values of their lists, the values of list tensors on the GPU -- seen
through results: a wrong entry would compute with another batch's sizes."""
import numpy as np
import pytest
import torch

from helpers import O
from blockedattention_b200 import _ops, blockAttention, blockAttnScores, blockAttnScoresHost, blockGEMM, blockSoftmax, clear_plan_cache

pytestmark = pytest.mark.gpu
PLANS, LISTS = 32, 256   # the bounds


def check_softmax(x, rows, cols, r, c):
    """blockSoftmax under the list arguments r, c gives the softmax of blocks rows x cols."""
    got = blockSoftmax(x, r, c).cpu()
    assert (got - O.block_softmax(x.cpu(), np.array(rows), np.array(cols))).abs().max() < 1e-6


@pytest.fixture()
def x(cuda_device):
    clear_plan_cache()
    return torch.randn((2, 24), generator=torch.Generator().manual_seed(0)).to(cuda_device)


def test_in_place_write_to_a_gpu_list_is_seen(cuda_device, x):
    r, c = (torch.tensor(t, device=cuda_device) for t in ([2, 3], [6, 4]))
    check_softmax(x, [2, 3], [6, 4], r, c)
    check_softmax(x, [2, 3], [6, 4], r, c)
    assert _ops.cached() == (1, 2)
    r[0], r[1], c[0], c[1] = 3, 2, 4, 6
    check_softmax(x, [3, 2], [4, 6], r, c)
    c.copy_(torch.tensor([6, 3])), r.copy_(torch.tensor([2, 4]))
    check_softmax(x, [2, 4], [6, 3], r, c)


def test_equal_values_share_a_plan(cuda_device, x):
    made = [lambda t: torch.tensor(t, device=cuda_device), lambda t: torch.tensor(t, device=cuda_device, dtype=torch.int32),
            lambda t: np.array(t), list, lambda t: torch.tensor(t), lambda t: torch.tensor([v for a in t for v in (a, -1)], device=cuda_device)[::2]]
    for as_list in made:
        check_softmax(x, [2, 3], [6, 4], as_list([2, 3]), as_list([6, 4]))
        assert _ops.cached()[0] == 1


def test_views_of_one_storage_are_different_lists(cuda_device, x):
    rows = torch.tensor([2, 4, 3], device=cuda_device)
    cols = torch.tensor([6, 3, 4], device=cuda_device)
    for _ in range(2):   # the same address, version, size and type, other strides
        check_softmax(x, [2, 3], [6, 4], rows[::2], cols[::2])
        check_softmax(x, [2, 4], [6, 3], rows[:2], cols[:2])


def test_lists_made_in_inference_mode_are_read_every_time(cuda_device, x):
    with torch.inference_mode():   # they have no version that would move
        r, c = (torch.tensor(t, device=cuda_device) for t in ([2, 3], [6, 4]))
    check_softmax(x, [2, 3], [6, 4], r, c)
    with torch.inference_mode():
        r.copy_(torch.tensor([3, 2])), c.copy_(torch.tensor([4, 6]))
    check_softmax(x, [3, 2], [4, 6], r, c)


def test_freed_lists_and_the_bounds(cuda_device):
    clear_plan_cache()
    kept = []
    for i in range(LISTS // 2 + 20):   # two lists a call; most are freed at once and their memory comes back
        rows, cols = [1 + i % 7, 2], [3, 1 + i % 11]
        D = int(np.dot(rows, cols))
        x = torch.randn((1, D), device=cuda_device)
        r, c = torch.tensor(rows, device=cuda_device), torch.tensor(cols, device=cuda_device)
        check_softmax(x, rows, cols, r, c)
        if i % 3 == 0:
            kept.append((x, rows, cols, r, c))
        plans, lists = _ops.cached()
        assert plans <= PLANS and lists <= LISTS
    assert _ops.cached() == (PLANS, LISTS)
    for args in kept:
        check_softmax(*args)
    clear_plan_cache()
    assert _ops.cached() == (0, 0)
    check_softmax(*kept[0])


def test_eviction_between_forward_and_backward(cuda_device):
    dev, d = cuda_device, 64
    n, kl = np.array([20, 100]), np.array([64, 64])
    g = torch.Generator(device=dev).manual_seed(0)
    q, k, v = ((torch.randn((2, int(n.sum()) * d), generator=g, device=dev) * 0.3).half() for _ in range(3))
    grads = []
    for evict in (False, True):
        leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
        clear_plan_cache()
        outs = [blockGEMM(*leaves[:2], None, None, None, n, n, kl), blockAttnScores(*leaves[:2], n, n, kl, scale=0.1),
                blockAttention(*leaves, n, n, scale=0.1, d=d)]
        outs.append(blockSoftmax(outs[0], n, n))
        if evict:
            for i in range(PLANS + 3):
                blockSoftmax(torch.zeros((1, 3 + i), device=dev), [1], [3 + i])
            clear_plan_cache()
        grads.append(torch.autograd.grad(sum(o.float().square().sum() for o in outs), leaves))
    assert all(torch.equal(a, b) for a, b in zip(*grads))


def test_host_pipe_follows_the_values_of_its_lists(cuda_device):
    # lists of one storage, and a numpy array written to behind its tensor's back
    g = torch.Generator().manual_seed(3)
    base = torch.tensor([30, 50, 10])
    a = np.array([30, 50])
    alias = torch.from_numpy(a)

    def check(n, lists):
        n = np.array(n)
        kl = np.full(len(n), 64)
        q, k = (torch.randn((2, int(n.sum()) * 64), generator=g).half() for _ in range(2))
        got = blockAttnScoresHost(q, k, lists, lists, kl, scale=0.125, device=cuda_device)
        torch.cuda.synchronize()
        assert (got.float() - O.block_scores(q, k, n, n, kl, scale=0.125)).abs().max() < 2e-3

    check([30, 50], base[:2])
    check([30, 10], base[::2])
    check([30, 50], alias)
    a[:] = 70, 20
    check([70, 20], alias)
