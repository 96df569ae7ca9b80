"""GPU: the operators and the process's other Python threads."""
import threading
import time

import numpy as np
import pytest
import torch

from blockedattention_b200 import (blockAttention, blockAttnScoresHost, blockGEMM, blockSoftmax, check_plans,
                                   clear_plan_cache)

pytestmark = pytest.mark.gpu
BUSY = 0.3  # seconds of queued work that a call has to wait for


def longest_stall(dev, call):
    """``call`` in a thread behind BUSY seconds of work on its stream; the longest time the main thread stood still."""
    ended, result = threading.Event(), []

    def run():
        try:
            t = time.perf_counter()
            result.append(call())
            torch.cuda.current_stream(dev).synchronize()
            result.append(time.perf_counter() - t)
        finally:
            ended.set()

    torch.cuda.synchronize()
    torch.cuda._sleep(int(BUSY * 1.9e9))  # (cycles)
    thread = threading.Thread(target=run)
    worst, last = 0.0, time.perf_counter()
    thread.start()
    while not ended.is_set():
        time.sleep(0.001)
        now = time.perf_counter()
        worst, last = max(worst, now - last), now
    thread.join()
    assert len(result) == 2 and result[1] > BUSY / 2, "the call did not have to wait"
    return worst


@pytest.mark.parametrize("what", ["new GPU list", "list made in inference mode", "new plan", "check_plans", "eviction"])
def test_a_waiting_call_does_not_stop_other_threads(cuda_device, what):
    dev = cuda_device
    rows, cols = [40, 300], [30, 70]
    x = torch.randn((2, 40 * 30 + 300 * 70), device=dev)
    clear_plan_cache()
    call = lambda: blockSoftmax(x, np.array(rows), np.array(cols))
    if what == "new GPU list":
        r, c = (torch.tensor(t, device=dev) for t in (rows, cols))
        call = lambda: blockSoftmax(x, r, c)
    elif what == "list made in inference mode":
        with torch.inference_mode():
            r, c = (torch.tensor(t, device=dev) for t in (rows, cols))
        call = lambda: blockSoftmax(x, r, c)
        call()
    elif what == "check_plans":
        call()
        call = check_plans
    elif what == "eviction":   # releasing a plan's tables waits for the device
        call()
        call = clear_plan_cache
    assert longest_stall(dev, call) < BUSY / 3


def test_threads_and_streams_share_the_caches(cuda_device):
    # the same and different batches from several threads, each on a stream of its own, forward and backward, with more
    # batches than plans are kept
    dev, d, H = cuda_device, 64, 2
    batches = [np.array([20 + i, 90 - i, 5]) for i in range(40)]

    def inputs(n, seed):
        g = torch.Generator(device=dev).manual_seed(seed)
        return [torch.randn((H, int(n.sum()) * d), generator=g, device=dev).half().requires_grad_(True) for _ in range(3)]

    def work(i):
        n = batches[i]
        q, k, v = inputs(n, i)
        lists = torch.tensor(n, device=dev) if i % 2 else n
        s = blockGEMM(q, k, None, None, None, lists, lists, np.full(3, d), scale=0.125)
        p = blockSoftmax(s, lists, lists)
        o = blockAttention(q, k, v, lists, lists, scale=0.125, d=d)
        grads = torch.autograd.grad((p.float().square().sum() + o.float().sum(),), (q, k, v))
        return [t.detach().clone() for t in (s, p, o) + grads]

    want = [work(i) for i in range(len(batches))]
    torch.cuda.synchronize()
    clear_plan_cache()
    failures = []

    def run(t):
        try:
            with torch.cuda.stream(torch.cuda.Stream(dev)):
                for j in range(2 * len(batches)):
                    i = (7 * j + 3 * t) % len(batches) if t % 2 else j % len(batches)
                    got = work(i)
                    torch.cuda.current_stream().synchronize()
                    if not all(torch.equal(a, b) for a, b in zip(got, want[i])):
                        failures.append((t, i))
        except Exception as e:  # noqa: BLE001 -- handed to the main thread
            failures.append((t, repr(e)))

    threads = [threading.Thread(target=run, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures[:5]


def test_host_pipe_from_several_streams_and_threads(cuda_device):
    # calls on one batch share its device buffers: a call from another stream must not overtake the one before
    n, kl, H = np.array([300, 200, 40]), np.full(3, 64), 8
    g = torch.Generator().manual_seed(0)
    ins = [[torch.randn((H, int(n.sum()) * 64), generator=g).half().pin_memory() for _ in range(2)] for _ in range(4)]

    def call(i):
        return blockAttnScoresHost(*ins[i], n, n, kl, scale=0.125, device=cuda_device)

    want = []
    for i in range(4):
        want.append(call(i))
        torch.cuda.synchronize()
    wrong = []

    def run(t):
        streams = [torch.cuda.Stream(cuda_device) for _ in range(4)]
        for _ in range(5):
            got = []
            for i, s in enumerate(streams):
                with torch.cuda.stream(s):
                    got.append(call(i))
            for i, s in enumerate(streams):
                s.synchronize()
                if not torch.equal(got[i], want[i]):
                    wrong.append((t, i))

    run("alone")
    threads = [threading.Thread(target=run, args=(t,)) for t in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:5]
