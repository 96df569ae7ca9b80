"""Python surface: ``blockGEMM`` and ``blockSoftmax`` with the upstream
signatures (``blockedAttention/apply.py:6-11`` and ``:27-30``), plus the fused
``blockAttnScores``.

Differences from upstream, all at the boundary:

* keyword-only extensions ``scale``, ``out_dtype`` and ``softmax`` (defaults
  reproduce upstream behaviour: no scale, output dtype = input dtype, separate
  softmax call);
* lists/offsets are read to the host once per distinct list tensor (kept
  alive while remembered, so an address cannot come back with other values)
  and the plan is cached under the list *values*, where upstream synchronises
  seven to eleven times per call;
* the shape checks upstream leaves to ``assert`` raise ``RuntimeError``;
* ``blockSoftmax`` passes its arguments by name, so ``srcAccum`` reaches the
  offsets parameter (upstream ``apply.py:41`` hands it to ``rowList``);
* autograd: both operators record the same backward as upstream
  (``csrc/sparseBlockedAttention.cpp:52-72``: two blocked GEMMs with permuted
  lists, offsets and transposition flags; ``:103-114``: the softmax backward
  kernel); the fused ``blockAttnScores`` chains the two.  As upstream, the
  operand gradients are laid out (m, k) / (n, k) row-major whatever the
  forward transposition flags were.
"""
from __future__ import annotations

import threading
from collections import OrderedDict
from contextlib import contextmanager
from typing import Optional

import torch

from . import _lib as L
from . import _ops
from .plan import GemmPlan, _host_i64



@contextmanager
def _untraced():
    state = torch._C._get_tracing_state()
    torch._C._set_tracing_state(None)
    try:
        yield
    finally:
        torch._C._set_tracing_state(state)


class _Traced(torch.autograd.Function):
    """An operator call as ``torch.jit.trace`` records it: one node with the call's operands as inputs, whose forward runs
    on every replay.  Lists, offsets and options are constants of the trace."""

    @staticmethod
    def forward(ctx, name, rest, *operands):
        with _untraced(), torch.enable_grad():
            ctx.operands = [t.detach().requires_grad_(t.requires_grad) for t in operands]
            ctx.result = getattr(_ops, name)(*ctx.operands, *rest)
            result = ctx.result.detach()
        if torch.jit.is_tracing():   # the tracer must have seen the result being made
            seen = torch.empty(0, dtype=result.dtype, device=result.device)
            with _untraced():
                seen.data = result
            result = seen
        return result

    @staticmethod
    def backward(ctx, grad):
        wanted = [t for t in ctx.operands if t.requires_grad]
        grads = iter(torch.autograd.grad(ctx.result, wanted, grad))
        return (None, None) + tuple(next(grads) if t.requires_grad else None for t in ctx.operands)


def _traced(name, operands, args):
    """Called by the native operators instead of running when the tracer is on."""
    if name == "softmax" and args[-1] is not None:   # in place or into a given tensor: nothing to record
        with _untraced():
            return _ops.softmax(*args)
    return _Traced.apply(name, args[operands:], *args[:operands])


_ops.setup(_host_i64, L.BlkError, _traced)

# The host pipes of blockAttnScoresHost, least recently used first, under the values of their lists.  (Plans and GPU lists
# of the operators are remembered by the native code.)
_CACHE: "OrderedDict[tuple, object]" = OrderedDict()
_CACHE_MAX = 32
_CACHE_LOCK = threading.Lock()


def _cached(key, build):
    with _CACHE_LOCK:
        found = _CACHE.get(key)
        if found is not None:
            _CACHE.move_to_end(key)
            return found
    made = build()
    dropped = []   # released after the lock, and only for the table: a queued step may still hold one
    with _CACHE_LOCK:
        found = _CACHE.setdefault(key, made)
        _CACHE.move_to_end(key)
        while len(_CACHE) > _CACHE_MAX:
            dropped.append(_CACHE.popitem(last=False))
    return found


def clear_plan_cache() -> None:
    """Forgets every cached plan and list (plans still referenced elsewhere stay usable)."""
    _ops.clear()
    with _CACHE_LOCK:
        dropped = list(_CACHE.values())
        _CACHE.clear()
    del dropped


def check_plans() -> None:
    """Synchronises the current stream of every cached plan's device and raises ``BlkError``
    (``BLK_ERR_TIMEOUT``) if a kernel of one of them gave up a bounded device-side wait since the last check --
    the result of that call is then incomplete.  ``BLK_CHECK=1`` in the environment does this after every run."""
    _ops.check()
    with _CACHE_LOCK:
        pipes = list(_CACHE.values())
    for plan in pipes:
        inner = getattr(plan, "plan", plan)   # a host pipe wraps its plan
        if getattr(inner, "device", None) is not None:
            inner.check()


def blockGEMM(mat1: torch.Tensor, mat2: torch.Tensor,
              mat1Accum: Optional[torch.Tensor] = None, mat2Accum: Optional[torch.Tensor] = None,
              outAccum: Optional[torch.Tensor] = None,
              MList: Optional[torch.Tensor] = None, NList: Optional[torch.Tensor] = None,
              KList: Optional[torch.Tensor] = None,
              transpose1: Optional[bool] = False, transpose2: Optional[bool] = False,
              *, scale: float = 1.0, out_dtype: Optional[torch.dtype] = None,
              softmax: bool = False) -> torch.Tensor:
    """Varlen blocked GEMM over a packed, head-major batch.

    ``mat1 -> (H, sum m_s*k_s)``, ``mat2 -> (H, sum n_s*k_s)``, result
    ``(H, sum m_s*n_s)`` with ``out_s = mat1_s @ mat2_s^T``.  Give either the
    three offset tensors (``mat1Accum = (0, m1*k1, m1*k1+m2*k2, ...)`` and so
    on) or the three lists (``MList = (m1, m2, ...)``), or both.
    ``transpose1``: mat1_s is stored (k, m); ``transpose2``: mat2_s is stored
    (k, n).  Any leading shape of mat1 flattens to H.
    """
    return _ops.gemm(mat1, mat2, mat1Accum, mat2Accum, outAccum, MList, NList, KList, transpose1, transpose2, scale,
                     out_dtype, softmax)


def blockSoftmax(src: torch.Tensor, rowList: torch.Tensor, colList: torch.Tensor,
                 srcAccum: Optional[torch.Tensor] = None, *, scale: float = 1.0,
                 out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Row softmax (last dim) of every packed block.

    ``src -> (H, sum rows_s*cols_s)``, result has the same shape; ``rowList =
    (rows_1, rows_2, ...)``, ``colList = (cols_1, ...)``; ``srcAccum = (0,
    rows_1*cols_1, ...)`` is optional.  ``out=src`` runs in place.
    """
    return _ops.softmax(src, rowList, colList, srcAccum, scale, out)


def blockAttnScores(q: torch.Tensor, k: torch.Tensor, MList, NList, KList, scale: float = 1.0,
                    out_dtype: Optional[torch.dtype] = None) -> torch.Tensor:
    """``softmax_rows(scale * Q_s K_s^T)`` for every segment in one pass: the
    fused form of ``blockSoftmax(blockGEMM(q, k, ...), MList, NList)``; the raw
    scores are never written to memory."""
    return _ops.gemm(q, k, None, None, None, MList, NList, KList, False, False, scale, out_dtype, True)


def blockAttention(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, MList, NList, scale: float = 1.0,
                   d: Optional[int] = None) -> torch.Tensor:
    """``softmax_rows(scale * Q_s K_s^T) V_s`` per segment: ``q -> (H, sum m_s*d)``, ``k, v -> (H, sum n_s*d)``, result
    ``(H, sum m_s*d)``, all packed head-major.  With 16-bit inputs and ``d`` 64 or 128 the batch runs as one kernel
    that never stores the probabilities (the pack kernel when every segment has at most 64 rows and columns and
    ``d = 64``, the tcgen05 attention kernel otherwise); any other batch is the composition
    ``blockGEMM(blockAttnScores(q, k), v, transpose2=True)`` of the two operators.  Carries autograd history: the
    fused batches have backward kernels of their own, which recompute the probabilities (from saved row logarithms for
    segments beyond 64 x 64); the composition differentiates through its operators."""
    return _ops.attention(q, k, v, MList, NList, scale, d)


def blockAttentionTokenMajor(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, nList, scale: float = 1.0) -> torch.Tensor:
    """Self-attention over a batch of graphs in the layout attention layers keep their activations in:
    ``q, k, v -> (sum n_s, H, d)`` (the nodes of all graphs in batch order), ``d`` 64 or 128, result of the same
    shape: ``out[rows of s] = softmax(scale * Q_s K_s^T) V_s`` per graph and head.  One kernel, no permuted copies,
    no probabilities in memory; graphs of any size, 16-bit inputs.  Forward only."""
    return _ops.attention_token_major(q, k, v, nList, scale)


def blockAttnScoresTokenMajor(q: torch.Tensor, k: torch.Tensor, nList, scale: float = 1.0,
                              out_dtype: Optional[torch.dtype] = None, softmax: bool = True) -> torch.Tensor:
    """``blockAttnScores`` for the layout attention inputs usually arrive in: ``q, k -> (sum n_s, H, d)``, the tokens
    of all segments in batch order.  The operands are read in place through strided tensor maps -- no permuted copy
    into head-major strips is made -- and the result is the packed head-major ``(H, sum n_s^2)`` buffer of
    ``blockAttnScores``.  Needs 16-bit inputs and ``d`` a multiple of 8 (16-byte rows for the tensor maps); with ``d = 32`` a batch
    with hundreds of segments of at most 64 tokens is refused (those run on a kernel that reads packed strips only).
    Forward only."""
    return _ops.scores_token_major(q, k, nList, scale, out_dtype, softmax)


class _HostPipe:
    """Device-side staging of ``blockAttnScoresHost`` for one (lists, H, dtypes, device): a plan for a group of
    heads, two sets of device buffers and three streams (copy in, compute, copy out)."""

    def __init__(self, M, N, K, H, groups, dtype, odt, softmax, device):
        self.groups, self.Hg = groups, H // groups
        self.plan = GemmPlan(M, N, K, self.Hg, dtype, odt, False, False, softmax, device=device)
        p = self.plan
        self.bufs = [(torch.empty((self.Hg, p.Dm1), dtype=dtype, device=device),
                      torch.empty((self.Hg, p.Dm2), dtype=dtype, device=device),
                      torch.empty((self.Hg, p.Dout), dtype=odt, device=device)) for _ in range(2)]
        self.s_in, self.s_run, self.s_out = (torch.cuda.Stream(device=device) for _ in range(3))
        for t in (t for buffers in self.bufs for t in buffers):
            for s in (self.s_in, self.s_run, self.s_out):
                t.record_stream(s)     # allocated on the stream of the first call
        self.lock = threading.Lock()   # one call's steps are queued at a time
        self.idle = None               # event: the last call is through with the buffers


def blockAttnScoresHost(q: torch.Tensor, k: torch.Tensor, MList, NList, KList, scale: float = 1.0,
                        out: Optional[torch.Tensor] = None, out_dtype: Optional[torch.dtype] = None,
                        device=None, softmax: bool = True, head_groups: Optional[int] = None) -> torch.Tensor:
    """``blockAttnScores`` for operands and result that live in host memory.

    ``q -> (H, sum m_s*k_s)``, ``k -> (H, sum n_s*k_s)`` and the result ``(H, sum m_s*n_s)`` are host tensors
    (pinned memory makes the copies asynchronous).  The heads are processed in ``head_groups`` groups (default:
    one head per group, at most eight groups): while group g is computed, group g+1 is copied to the device and
    the result of group g-1 is copied back, so the transfer of the result and the arithmetic hide behind the
    transfer of the operands.  The call is ordered after work already queued on the current stream and the
    current stream waits for the last copy: synchronise it before reading ``out`` on the host.
    """
    for name, t in (("q", q), ("k", k)):
        if not isinstance(t, torch.Tensor) or t.is_cuda:
            raise RuntimeError(f"{name} must be a host tensor")
        if not t.is_contiguous():
            raise RuntimeError(f"{name} must be contiguous Tensor")
    if q.dtype != k.dtype:
        raise RuntimeError("q and k must have the same dtype")
    dev = torch.device(device) if device is not None else torch.device("cuda", torch.cuda.current_device())
    odt = out_dtype if out_dtype is not None else q.dtype
    M, N, K = _host_i64(MList), _host_i64(NList), _host_i64(KList)
    Dm1, Dm2, Dout = int((M * K).sum()), int((N * K).sum()), int((M * N).sum())
    if Dm1 <= 0 or q.numel() % Dm1 or k.numel() != (q.numel() // Dm1) * Dm2:
        raise RuntimeError("q / k do not match the packed extents of the lists")
    H = q.numel() // Dm1
    groups = head_groups if head_groups is not None else next(g for g in range(min(H, 8), 0, -1) if H % g == 0)
    if groups < 1 or H % groups:
        raise RuntimeError(f"head_groups = {groups} does not divide H = {H}")
    if out is None:
        out = torch.empty((H, Dout), dtype=odt).pin_memory()
    elif out.is_cuda or not out.is_contiguous() or out.dtype != odt or out.numel() != H * Dout:
        raise RuntimeError("out must be a contiguous host tensor of the output dtype with H*Dout elements")
    key = ("hostpipe", M.tobytes(), N.tobytes(), K.tobytes(), H, groups, q.dtype, odt, bool(softmax), str(dev))
    pipe = _cached(key, lambda: _HostPipe(M, N, K, H, groups, q.dtype, odt, bool(softmax), dev))
    Hg = pipe.Hg
    qv, kv, ov = q.reshape(H, Dm1), k.reshape(H, Dm2), out.reshape(H, Dout)
    cur = torch.cuda.current_stream(dev)
    start = torch.cuda.Event()
    start.record(cur)
    with pipe.lock:
        for s in (pipe.s_in, pipe.s_run, pipe.s_out):
            s.wait_event(start)
            if pipe.idle is not None:   # (the call before may have come from another stream)
                s.wait_event(pipe.idle)
        ran = [None, None]     # per buffer set: event after the kernels that read its operands
        drained = [None, None]  # per buffer set: event after the copy that read its result
        for g in range(groups):
            b = g & 1
            dq, dk, do = pipe.bufs[b]
            rows = slice(g * Hg, (g + 1) * Hg)
            with torch.cuda.stream(pipe.s_in):
                if ran[b] is not None:
                    pipe.s_in.wait_event(ran[b])
                dq.copy_(qv[rows], non_blocking=True)
                dk.copy_(kv[rows], non_blocking=True)
                loaded = torch.cuda.Event()
                loaded.record(pipe.s_in)
            with torch.cuda.stream(pipe.s_run):
                pipe.s_run.wait_event(loaded)
                if drained[b] is not None:
                    pipe.s_run.wait_event(drained[b])
                pipe.plan.run(dq, dk, out=do, scale=scale)
                ran[b] = torch.cuda.Event()
                ran[b].record(pipe.s_run)
            with torch.cuda.stream(pipe.s_out):
                pipe.s_out.wait_event(ran[b])
                ov[rows].copy_(do, non_blocking=True)
                drained[b] = torch.cuda.Event()
                drained[b].record(pipe.s_out)
        pipe.idle = drained[(groups - 1) & 1]
    for ev in drained:
        if ev is not None:
            cur.wait_event(ev)
    return out
