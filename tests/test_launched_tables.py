"""CPU: batches whose kernel runs a list of its own -- the streams of ``blk_scores_umma.cu``, the 128 x 128 tiles of the fp32
kernel -- hold that list to the same: every output element belongs to one item of what is launched."""
import numpy as np
import pytest
import torch

from blockedattention_b200.plan import GemmPlan


@pytest.mark.parametrize("forced", [False, True])
@pytest.mark.parametrize("softmax", [False, True])
def test_streams_take_the_tcgen05_items_costliest_first(monkeypatch, forced, softmax):
    rs = np.random.RandomState(3 + softmax)
    if forced:
        monkeypatch.setenv("BLK_UMMA_STREAMS", "1")
        n, m, H = rs.randint(1, 400, 200), rs.randint(1, 300, 200), 2
        K = rs.choice([16, 48, 64] if softmax else [16, 48, 64, 96, 128], 200)
    else:  # a batch that is large enough by itself
        n = rs.randint(100, 2000, 20)
        m, K, H = n, np.full(20, 64), 4
    plan = GemmPlan(m, n, K, H, torch.bfloat16, softmax=softmax)
    items, run = plan.table("umma_items"), plan.table("stream_items")
    assert run.size == items.size > 0
    assert np.array_equal(np.sort(run.view("V48")), np.sort(items.view("V48")))
    assert (run["nch"] == 0).all()                       # whole rows: the kernel knows no column ranges
    cost = (run["N"].astype(np.int64) + 63) // 64 * 2 + (run["K"] > 64)
    assert (np.diff(cost) <= 0).all()


@pytest.mark.parametrize("kw", [{}, dict(transpose1=True), dict(transpose2=True), dict(softmax=True)])
def test_fp32_tiles_of_both_sizes_cover_every_element_once(kw):
    rs = np.random.RandomState(4)
    m = np.concatenate([rs.randint(1, 64, 30), rs.randint(64, 700, 40)])
    n = np.concatenate([rs.randint(1, 64, 30), rs.randint(64, 700, 40)])
    plan = GemmPlan(m, n, rs.randint(1, 100, 70), 2, torch.float32, **kw)
    big, rest = plan.table("simt_big"), plan.table("simt_rest")
    assert big.size and rest.size and plan.summary["launches"] == 2 + bool(kw.get("softmax"))
    cover = [np.zeros((a, b), np.int32) for a, b in zip(m, n)]
    for items, t in ((big, 128), (rest, 64)):
        for it in items:
            assert it["ntn"] == 1
            cover[it["seg"]][it["tm"] * t:(it["tm"] + 1) * t, it["tn"] * t:(it["tn"] + 1) * t] += 1
    assert all((c == 1).all() for c in cover)


def test_other_batches_run_the_first_lists():
    plan = GemmPlan([300, 40], [200, 70], [64, 64], 2, torch.float16)
    assert plan.table("umma_items").size and not plan.table("stream_items").size
    plan = GemmPlan([300, 40], [200, 70], [64, 64], 2, torch.float32)
    assert plan.table("simt_items").size and not plan.table("simt_big").size and not plan.table("simt_rest").size
