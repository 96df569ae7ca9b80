"""The calls that performance is measured on: what a program that uses this package has it do, at the sizes and data
types of the package's own workloads (``blockedattention_b200/synth.py``) and around them.

A case is a dict of plain values.  ``op`` names the call, ``dist``/``lo``/``hi`` the distribution of the segment sizes
(drawn from ``sizes``, so a case always has the same segments), ``segments``/``heads``/``d``/``dtype`` the batch and
``lists`` how the program holds the segment sizes: int64 tensors on the GPU, as callers of the two original operators
do, or numpy arrays, as a data loader leaves them.  Every call goes through the functional entry points.

    chain            blockSoftmax(blockGEMM(q, k)): the two operators as a script calls them
    chain_train      the same with autograd: gradients of q and k
    scores           blockAttnScores: both in one call
    forward          blockAttnScores, then the product with the values through blockGEMM(transpose2=True)
    attention        blockAttention, packed head-major strips
    attention_tokens blockAttentionTokenMajor, (tokens, heads, d) tensors in and out
    attention_train  blockAttention with autograd: gradients of q, k and v
    gemm             blockGEMM alone
    softmax          blockSoftmax alone
    softmax_train    blockSoftmax with autograd
"""
import math

import numpy as np
import torch

import blockedattention_b200 as ba

_DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}
_BYTES = {"fp16": 2, "bf16": 2, "fp32": 4}
_TRAIN = ("chain_train", "attention_train", "softmax_train")


def _case(name, op, segments, dist, lo, hi, heads, d, dtype, lists, out="", kdist="d", sizes=0):
    return {"name": name, "op": op, "segments": segments, "dist": dist, "lo": lo, "hi": hi, "heads": heads, "d": d,
            "dtype": dtype, "out": out or dtype, "kdist": kdist, "lists": lists, "sizes": sizes}


def listed():
    return [
        # a script's first call and a unit test's batch: 32 small fp32 segments, one head; all latency
        _case("script_chain", "chain", 32, "uniform", 4, 32, 1, 32, "fp32", "cuda"),
        # one inference request: 16 molecular graphs through one attention layer
        _case("request_attention", "attention_tokens", 16, "graphs", 2, 64, 8, 64, "fp16", "numpy"),
        # a large molecular batch, attention probabilities wanted
        _case("molecular_scores", "scores", 4096, "graphs", 2, 128, 8, 64, "fp16", "cuda"),
        # a training step's attention over a molecular mini-batch
        _case("molecular_train", "attention_train", 1024, "graphs", 2, 128, 8, 64, "fp16", "cuda"),
        # blocked products of unrelated sizes, fp16 in and fp32 out
        _case("general_gemm", "gemm", 2048, "pair", 1, 256, 1, 128, "fp16", "cuda", out="fp32", kdist="steps16"),
        # sizes over two decades: the batch the throughput is quoted on
        _case("long_tail_scores", "scores", 512, "log", 16, 2048, 4, 64, "bf16", "numpy"),
        # the second operator alone, over the score buffer of that batch
        _case("long_tail_softmax", "softmax", 512, "log", 16, 2048, 4, 64, "bf16", "cuda"),
        # both operators with autograd, as a layer written on the original interface trains
        _case("long_tail_chain_train", "chain_train", 128, "log", 16, 2048, 4, 64, "bf16", "cuda"),
        # a whole layer's forward with the probabilities kept: P, then P V
        _case("full_forward", "forward", 1024, "uniform", 64, 512, 16, 128, "bf16", "cuda"),
        # the same layer at inference, probabilities not wanted, activations as the layer holds them
        _case("full_attention", "attention_tokens", 1024, "uniform", 64, 512, 16, 128, "bf16", "numpy"),
        # and in training
        _case("full_train", "attention_train", 256, "uniform", 64, 512, 16, 128, "bf16", "cuda"),
        # few large products with long contractions
        _case("large_k", "gemm", 64, "square", 1024, 2048, 1, 4096, "fp16", "cuda", kdist="octaves"),
    ]


def _sizes(case):
    """(M, N, K) of every segment."""
    rs = np.random.RandomState(case["sizes"])
    S, lo, hi = case["segments"], case["lo"], case["hi"]
    if case["dist"] == "graphs":      # node counts of molecular graphs
        m = np.clip(np.rint(rs.normal(25.0, 10.0, size=S)), lo, hi)
    elif case["dist"] == "log":
        m = np.clip(np.rint(np.exp(rs.uniform(math.log(lo), math.log(hi), size=S))), lo, hi)
    else:
        m = rs.randint(lo, hi + 1, size=S)
    n = rs.randint(lo, hi + 1, size=S) if case["dist"] == "pair" else m
    d = case["d"]
    if case["kdist"] == "steps16":
        k = rs.choice([x for x in (16, 32, 48, 64, 96, 128) if x <= d], size=S)
    elif case["kdist"] == "octaves":
        k = rs.choice([d // 4, d // 2, d], size=S)
    elif case["kdist"] == "any":
        k = rs.randint(16, d + 1, size=S)
    else:
        k = np.full(S, d)
    return tuple(np.asarray(x, dtype=np.int64) for x in (m, n, k))


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["chain", "chain_train", "scores", "scores", "forward", "attention", "attention_tokens",
                     "attention_train", "attention_train", "gemm", "gemm", "softmax", "softmax_train"])
    dtype = rng.choice(["fp16", "bf16"])
    out, kdist, d = dtype, "d", rng.choice([64, 128])
    heads = rng.choice([1, 2, 4, 8, 16])
    dist, lo, hi = rng.choice([("graphs", 2, 128), ("uniform", 1, log(32, 512)), ("log", 16, log(128, 2048))])
    if op in ("chain", "chain_train", "scores", "forward"):
        d = rng.choice([32, 64, 64, 128])
    if op in ("chain", "chain_train", "softmax", "softmax_train") and rng.random() < 0.3:
        dtype = out = "fp32"
    if op == "gemm":
        heads = rng.choice([1, 1, 4])
        if rng.random() < 0.3:
            dist, lo, hi, d, kdist = "square", 256, log(512, 2048), 8 * log(128, 512), rng.choice(["d", "octaves"])
        else:
            dist, lo, hi, d, kdist = "pair", 1, log(32, 512), 128, rng.choice(["steps16", "steps16", "any"])
        dtype = rng.choice(["fp16", "fp16", "bf16", "fp32"])
        out = "fp32" if rng.random() < 0.5 else dtype
    case = {"op": op, "segments": log(4, 4096), "dist": dist, "lo": lo, "hi": hi, "heads": heads, "d": d, "dtype": dtype,
            "out": out, "kdist": kdist, "lists": rng.choice(["cuda", "numpy"]), "sizes": rng.randrange(1, 1 << 20)}
    most = max(_cost(c) for c in listed())
    while _cost(case) > most:
        case["segments"] = max(1, case["segments"] * 2 // 3)
    return case


def _cost(case):
    """Seconds that a pass cannot do without, roughly: only for keeping draws below the largest listed case."""
    w = work(case)
    return max(w["bytes"] / 6.5e12, w["flops"] / (6e13 if case["dtype"] == "fp32" else 1.6e15))


def _made(case, seed, shape, std, dtype, uniform=False):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = torch.empty(shape, dtype=torch.float32, device="cuda")
    x = x.uniform_(-1.0, 1.0, generator=g) if uniform else x.normal_(0.0, std, generator=g)
    return x.to(dtype)


def prepare(case, seed):
    op, H, d, dt = case["op"], case["heads"], case["d"], _DTYPES[case["dtype"]]
    M, N, K = _sizes(case)
    as_lists = (lambda x: torch.from_numpy(x).cuda()) if case["lists"] == "cuda" else (lambda x: x)
    s = {"op": op, "scale": 1.0 / math.sqrt(d), "out": _DTYPES[case["out"]],
         "M": as_lists(M), "N": as_lists(N), "K": as_lists(K), "D": as_lists(np.full_like(M, d)), "d": d}

    def made(k, shape, std=1.0, uniform=False):
        return _made(case, seed * 8 + k, shape, std, dt, uniform)

    rows_q, rows_k, cells = int(M.sum()), int(N.sum()), int((M * N).sum())
    if op.startswith("softmax"):
        s["x"] = made(0, (H, cells), 2.0)
        if op in _TRAIN:
            s["x"].requires_grad_(True)
            s["g"] = made(1, (H, cells))
        return s
    tokens = op == "attention_tokens"
    uniform = op == "gemm"
    # the two operators take no scale: their callers fold it into q
    fold = s["scale"] if op.startswith("chain") else 1.0
    s["q"] = made(0, (rows_q, H, d) if tokens else (H, int((M * K).sum())), fold, uniform)
    s["k"] = made(1, (rows_k, H, d) if tokens else (H, int((N * K).sum())), 1.0, uniform)
    if op in ("forward", "attention", "attention_tokens", "attention_train"):
        s["v"] = made(2, (rows_k, H, d) if tokens else (H, rows_k * d))
    if op in _TRAIN:
        s["g"] = made(3, (H, cells if op == "chain_train" else rows_q * d))
        for name in ("q", "k", "v"):
            if name in s:
                s[name].requires_grad_(True)
    return s


def run(s):
    op, M, N, K = s["op"], s["M"], s["N"], s["K"]
    if op == "gemm":
        return ba.blockGEMM(s["q"], s["k"], None, None, None, M, N, K, out_dtype=s["out"])
    if op == "softmax":
        return ba.blockSoftmax(s["x"], M, N)
    if op == "softmax_train":
        p = ba.blockSoftmax(s["x"], M, N)
        return (p.detach(),) + torch.autograd.grad(p, (s["x"],), s["g"])
    if op == "chain":
        return ba.blockSoftmax(ba.blockGEMM(s["q"], s["k"], None, None, None, M, N, K), M, N)
    if op == "chain_train":
        p = ba.blockSoftmax(ba.blockGEMM(s["q"], s["k"], None, None, None, M, N, K), M, N)
        return (p.detach(),) + torch.autograd.grad(p, (s["q"], s["k"]), s["g"])
    if op == "scores":
        return ba.blockAttnScores(s["q"], s["k"], M, N, K, scale=s["scale"])
    if op == "forward":
        p = ba.blockAttnScores(s["q"], s["k"], M, N, K, scale=s["scale"])
        return p, ba.blockGEMM(p, s["v"], None, None, None, M, s["D"], N, False, True)
    if op == "attention":
        return ba.blockAttention(s["q"], s["k"], s["v"], M, N, scale=s["scale"], d=s["d"])
    if op == "attention_tokens":
        return ba.blockAttentionTokenMajor(s["q"], s["k"], s["v"], M, scale=s["scale"])
    o = ba.blockAttention(s["q"], s["k"], s["v"], M, N, scale=s["scale"], d=s["d"])
    return (o.detach(),) + torch.autograd.grad(o, (s["q"], s["k"], s["v"]), s["g"])


def work(case):
    """Every tensor the call is given read once, every tensor it returns written once; the products it cannot do
    without (an attention backward recomputes the scores: five products)."""
    op, H, e, eo = case["op"], case["heads"], _BYTES[case["dtype"]], _BYTES[case["out"]]
    M, N, K = (x.astype(np.float64) for x in _sizes(case))
    mk, nk, mn, d = float((M * K).sum()), float((N * K).sum()), float((M * N).sum()), case["d"]
    md, nd, mnk = float(M.sum()) * d, float(N.sum()) * d, float((M * N * K).sum())
    values, products = {
        "gemm": ((mk + nk) * e + mn * eo, mnk),
        "softmax": (2 * mn * e, 0.0),
        "softmax_train": (4 * mn * e, 0.0),                       # x, g in; p, dx out
        "chain": ((mk + nk + mn) * e, mnk),
        "chain_train": ((2 * mk + 2 * nk + 2 * mn) * e, 3 * mnk),  # q, k, g in; p, dq, dk out
        "scores": ((mk + nk + mn) * e, mnk),
        "forward": ((mk + nk + mn + nd + md) * e, mnk + mn * d),
        "attention": ((2 * md + 2 * nd) * e, 2 * mn * d),
        "attention_tokens": ((2 * md + 2 * nd) * e, 2 * mn * d),
        "attention_train": ((4 * md + 4 * nd) * e, 7 * mn * d),    # q, k, v, g in; o, dq, dk, dv out
    }[op]
    return {"bytes": H * values, "flops": 2.0 * H * products}


def tolerance(case):
    """One or a few roundings to the result's type; fp32 sums in another order."""
    if case["dtype"] == "fp32" or case["out"] == "fp32":
        return {"rel": 1e-5}
    return {"rel": 1e-2} if case["dtype"] == "bf16" else {"rel": 2e-3}
