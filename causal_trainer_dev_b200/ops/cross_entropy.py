"""Projection-fused ("cut") cross-entropy and its chunked / plain companions.

``cut_cross_entropy`` never materialises the ``[tokens, vocab]`` logits in the forward
pass: the LM-head GEMM runs on tcgen05 with an epilogue that reduces each 256-column
slab of a row to (max, sum-exp, target logit) while the tile is still in TMEM
(``csrc/gemm.cu``, EPI_CE_STATS); a small kernel merges the slabs into the row LSE and
the weighted NLL.  The backward pass recomputes logits chunk by chunk with the
``(softmax - onehot) * coef`` epilogue (EPI_CE_DLOGITS) into a bounded bf16 slab and feeds
two ordinary GEMMs (dHidden, dHead), so memory is O(chunk * vocab), not O(tokens * vocab).

Losses are *sums* (``nll_sum``, ``weight_sum``); the caller normalises globally, as
src/causal_trainer/training/steps.py:172 does.

Reference counterparts: pallas_cut_linear_cross_entropy
(src/causal_trainer/kernels/cut_cross_entropy.py:85-156, 225-278, 349-403, 828-960),
the chunked logits backend (src/causal_trainer/kernels/cross_entropy.py:99-189, 254-322)
and the XLA oracle (src/causal_trainer/kernels/fused_cross_entropy.py:64-109).
"""
from __future__ import annotations

import ctypes

import torch

from . import lib as _lib
from .gemm import gemm

SLAB = 256


def reference_cross_entropy(hidden, head, targets, weights):
    """fp32 oracle: returns (nll_sum, weight_sum).  head is [vocab, hidden]."""
    logits = hidden.float() @ head.float().t()
    lse = torch.logsumexp(logits, dim=-1)
    tgt = logits.gather(-1, targets.long().clamp_min(0)[:, None])[:, 0]
    w = weights.float()
    return ((lse - tgt) * w).sum(), w.sum()


def chunked_cross_entropy(hidden, head, targets, weights, token_budget: int = 4096):
    """Autograd-friendly chunked logits CE (the ``pallas``/``xla`` backends of the CLI).

    Walks row chunks of at most ``token_budget`` rows, skips chunks whose weights are all
    zero, and checkpoints each chunk so only one logits slab is alive at a time.
    """
    from torch.utils.checkpoint import checkpoint

    def one(h, t, w):
        logits = (h @ head.t()).float()
        lse = torch.logsumexp(logits, dim=-1)
        tgt = logits.gather(-1, t.long()[:, None])[:, 0]
        return ((lse - tgt) * w.float()).sum()

    total = hidden.new_zeros((), dtype=torch.float32)
    for start in range(0, hidden.shape[0], token_budget):
        w = weights[start:start + token_budget]
        if not bool((w != 0).any()):
            continue
        h, t = hidden[start:start + token_budget], targets[start:start + token_budget]
        if torch.is_grad_enabled() and (hidden.requires_grad or head.requires_grad):
            total = total + checkpoint(one, h, t, w, use_reentrant=False)
        else:
            total = total + one(h, t, w)
    return total, weights.float().sum()


def _target_words(targets: torch.Tensor) -> tuple[torch.Tensor, int]:
    """Target ids as the kernels read them: 32-bit words, every one (step 1) or, of 64-bit ids, the low one of two (step 2)."""
    if targets.dtype == torch.int64 and targets.is_contiguous():
        return targets, 2
    return targets.to(torch.int32).contiguous(), 1


def _device_scale(grad_scale, device) -> tuple[float, torch.Tensor | None]:
    """A factor of the gradients as (number, one fp32 element on the device or None).  A tensor on the host is a number: a copy
    to the device would wait for the stream, and cannot be captured."""
    if not isinstance(grad_scale, torch.Tensor):
        return grad_scale, None
    if grad_scale.device.type == "cpu":
        return grad_scale.reshape(()).to(torch.float32).item(), None
    return 1.0, grad_scale.reshape(()).to(device=device, dtype=torch.float32)


class _Scratch:
    """fp32 pieces of one allocation by their addresses (an allocation each costs more host time than a launch); it holds them
    while it lives."""

    def __init__(self, device, **counts: int):
        self.device = device
        self._whole = torch.empty(sum(counts.values()), dtype=torch.float32, device=device)
        at = self._whole.data_ptr()
        for name, count in counts.items():
            setattr(self, name, at)
            at += 4 * count


def _combine(L, work: _Scratch, slabs, tgt, step, vocab, w, scale, device_scale, lse, coef, start, rows):
    """Row statistics of the rows [start, start + rows) of a call (``work``: the slabs of these rows alone)."""
    p = ctypes.c_void_p
    code = L.ctb_ce_combine(p(work.pmax), p(work.psum), slabs, p(work.tlogit + 4 * start), p(tgt.data_ptr() + 4 * step * start),
                            step, vocab, p(w.data_ptr() + 4 * start), ctypes.c_float(scale), _lib.ptr(device_scale),
                            p(lse + 4 * start), p(coef + 4 * start), p(work.bn + start // 32 * 4), p(work.bw + start // 32 * 4),
                            rows, _lib.stream_ptr())
    _lib.check(code, "ctb_ce_combine")


def _sums(L, work: _Scratch, rows: int) -> tuple[torch.Tensor, torch.Tensor]:
    nll, wsum = (torch.empty((), dtype=torch.float32, device=work.device) for _ in range(2))
    code = L.ctb_ce_sums(ctypes.c_void_p(work.bn), ctypes.c_void_p(work.bw), _row_blocks(rows), _lib.ptr(nll), _lib.ptr(wsum),
                         _lib.stream_ptr())
    _lib.check(code, "ctb_ce_sums")
    return nll, wsum


def _row_blocks(rows: int) -> int:
    return (rows + 31) // 32          # partial sums of 32 rows each (csrc/elementwise.cu: CE_ROWS)


def cut_ce_forward(hidden, head, targets, weights, grad_scale: float | torch.Tensor = 1.0, exchange=None):
    """Returns (nll_sum, weight_sum, lse, coef); coef = weights * grad_scale for the backward.

    ``grad_scale`` may be a one-element device tensor (the reciprocal of a token count that was
    just all-reduced): it is applied on the device, so the caller never has to read it back.

    With ``exchange`` (vocabulary-parallel head: ``head`` holds this rank's vocabulary rows and
    ``targets`` are already relative to them, -1 elsewhere) the per-row statistics are combined
    across the tensor-parallel ranks inside ``exchange.ce_exchange``.
    """
    rows, d = hidden.shape
    vocab = head.shape[0]
    slabs = (vocab + SLAB - 1) // SLAB
    dev = hidden.device
    grad_scale, device_scale = _device_scale(grad_scale, dev)
    p = ctypes.c_void_p
    if exchange is None:
        work = _Scratch(dev, pmax=slabs * rows, psum=slabs * rows, tlogit=rows, bn=_row_blocks(rows), bw=_row_blocks(rows))
        parts = p(work.pmax), p(work.psum), p(work.tlogit)
    else:
        pmax, psum = (torch.empty((slabs, rows), dtype=torch.float32, device=dev) for _ in range(2))
        # (the exchange adds the ranks' target logits up: zero where a rank has none)
        tlogit = torch.zeros(rows, dtype=torch.float32, device=dev)
        parts = _lib.ptr(pmax), _lib.ptr(psum), _lib.ptr(tlogit)
    tgt, step = _target_words(targets)
    w = weights.to(torch.float32).contiguous()
    L = _lib.lib()
    from .gemm import _FLAG_SOURCES, _flag_args, _rotations, flag_source_of, in_gathered_buffer

    hit = flag_source_of(head) if _FLAG_SOURCES else None
    hit_a = flag_source_of(hidden) if _FLAG_SOURCES else None
    _, m_rotate = _rotations(None, hit_a, hidden, head, False, False, rows, vocab)
    code = L.ctb_ce_stats(_lib.ptr(hidden), _lib.ptr(head), rows, vocab, d, ctypes.c_long(hidden.stride(0)),
                          ctypes.c_long(head.stride(0)), _lib.ptr(tgt), step, *parts, *_flag_args(hit), *_flag_args(hit_a),
                          m_rotate, int(in_gathered_buffer(hidden, head)), None, ctypes.c_long(0), _lib.stream_ptr())
    _lib.check(code, "ctb_ce_stats")
    if exchange is not None:
        nll, wsum, lse, coef = exchange.ce_exchange(pmax, psum, slabs, tlogit, w, grad_scale)
        if device_scale is not None:
            coef.mul_(device_scale)
        return nll, wsum, lse, coef
    lse = torch.empty(rows, dtype=torch.float32, device=dev)
    coef = torch.empty(rows, dtype=torch.float32, device=dev)
    _combine(L, work, slabs, tgt, step, vocab, w, grad_scale, device_scale, lse.data_ptr(), coef.data_ptr(), 0, rows)
    return *_sums(L, work, rows), lse, coef


def cut_ce_backward(hidden, head, targets, lse, coef, *, chunk_rows: int = 4096, need_dhead: bool = True,
                    dhead_out: torch.Tensor | None = None, dhead_accumulate: bool = False, push=None):
    """Returns (dhidden [rows,d] bf16, dhead [vocab,d] or None).

    With ``push`` (vocabulary-parallel head) the partial ``dhidden`` tiles are reduce-scattered
    into the owners' receive buffers by the GEMM epilogue and ``dhidden`` is returned as None.
    """
    rows, d = hidden.shape
    vocab = head.shape[0]
    dev = hidden.device
    tgt, step = _target_words(targets)
    dhidden = torch.empty_like(hidden) if push is None else None
    dhead = None
    if need_dhead:
        dhead = dhead_out if dhead_out is not None else torch.empty((vocab, d), dtype=torch.bfloat16, device=dev)
    chunk_rows = min(chunk_rows, rows)
    if push is not None:
        if rows % 128:
            raise ValueError("the push epilogue needs a multiple of 128 rows")
        chunk_rows = max(128, chunk_rows // 128 * 128)
    slab = torch.empty((chunk_rows, vocab), dtype=torch.bfloat16, device=dev)
    L = _lib.lib()
    from .gemm import in_gathered_buffer

    gathered = int(in_gathered_buffer(hidden, head))
    first = True
    for start in range(0, rows, chunk_rows):
        n = min(chunk_rows, rows - start)
        h = hidden[start:start + n]
        g = slab[:n]
        code = L.ctb_ce_dlogits(_lib.ptr(h), _lib.ptr(head), _lib.ptr(g), n, vocab, d, ctypes.c_long(h.stride(0)),
                                ctypes.c_long(head.stride(0)), ctypes.c_long(g.stride(0)),
                                _lib.ptr(tgt[start:start + n]), step, _lib.ptr(lse[start:start + n]),
                                _lib.ptr(coef[start:start + n]), gathered, _lib.stream_ptr())
        _lib.check(code, "ctb_ce_dlogits")
        if push is None:
            gemm(g, head, b_mn=True, out=dhidden[start:start + n])              # dH = G @ W
        else:
            from .gemm import gemm_push

            gemm_push(g, head, push, b_mn=True, row_offset=start,
                      tiles_per_dest=(push.rows_per_rank // 128) * (-(-d // 256)))
        if need_dhead:
            gemm(g, h, a_mn=True, b_mn=True, out=dhead, accumulate=(dhead_accumulate or not first))  # dW += G^T H
        first = False
    return dhidden, dhead


# From this width on the logits of a chunk are kept in fp32 between the statistics and the gradient (forward and backward
# called as one): writing and reading an element again takes 8 bytes of memory, recomputing it 2 x width operations.
# Forward and backward, computed twice and kept, us: 2048 rows x 32000 x 512 325 and 311, x 768 393 and 361, 333 x 32000 x 1536
# 212 and 181, 8192 x 168384 x 1536 12700 and 11850, 4096 x 128256 x 4096 12700 and 10400.  Narrower ones are not measured.
KEEP_LOGITS_WIDTH = 512


def keeps_logits(rows: int, vocab: int, width: int, chunk_rows: int) -> bool:
    """Whether :func:`cut_ce_forward_backward` keeps the logits of a chunk (in plain, not in gathered buffers): then its slab
    holds 4 bytes for each, otherwise 2."""
    chunk_rows = min(chunk_rows, rows)
    return rows > 0 and width >= KEEP_LOGITS_WIDTH and vocab % 8 == 0 and (chunk_rows == rows or chunk_rows % 32 == 0)


def cut_ce_forward_backward(hidden, head, targets, weights, grad_scale: float | torch.Tensor = 1.0, *, chunk_rows: int = 4096,
                            need_dhead: bool = True, dhead_out: torch.Tensor | None = None, dhead_accumulate: bool = False,
                            keep_logits: bool = True):
    """:func:`cut_ce_forward` and :func:`cut_ce_backward` in one: ``(nll_sum, weight_sum, dhidden, dhead)``, the same bits.

    Row chunk by row chunk, so a chunk's fp32 logits can wait for their gradient (which takes their place) instead of being
    computed twice, where that is cheaper (:func:`keeps_logits`).  ``keep_logits=False``: the caller has no memory for them
    (chunk_rows x vocab x 4 bytes).  Their slab is the last that is allocated: where it finds no memory, half of it has to do,
    and while it lives nothing is allocated that could not do without."""
    rows, d = hidden.shape
    vocab = head.shape[0]
    from .gemm import in_gathered_buffer

    chunk_rows = min(chunk_rows, rows)

    def twice():
        nll, wsum, lse, coef = cut_ce_forward(hidden, head, targets, weights, grad_scale)
        dhidden, dhead = cut_ce_backward(hidden, head, targets, lse, coef, chunk_rows=chunk_rows, need_dhead=need_dhead,
                                         dhead_out=dhead_out, dhead_accumulate=dhead_accumulate)
        return nll, wsum, dhidden, dhead

    if not keep_logits or not keeps_logits(rows, vocab, d, chunk_rows) or in_gathered_buffer(hidden, head):
        return twice()
    dev = hidden.device
    scale, device_scale = _device_scale(grad_scale, dev)
    slabs = (vocab + SLAB - 1) // SLAB
    work = _Scratch(dev, pmax=slabs * chunk_rows, psum=slabs * chunk_rows, tlogit=rows, lse=rows, coef=rows,
                    bn=_row_blocks(rows), bw=_row_blocks(rows))
    tgt, step = _target_words(targets)
    w = weights.to(torch.float32).contiguous()
    dhidden = torch.empty_like(hidden)
    dhead = None
    if need_dhead:
        dhead = dhead_out if dhead_out is not None else torch.empty((vocab, d), dtype=torch.bfloat16, device=dev)
    try:
        slab = torch.empty((chunk_rows, vocab), dtype=torch.float32, device=dev)
    except torch.cuda.OutOfMemoryError:
        slab = None
    if slab is None:
        del work, dhidden, dhead
        return twice()
    L, ln, p = _lib.lib(), ctypes.c_long, ctypes.c_void_p
    for start in range(0, rows, chunk_rows):
        n = min(chunk_rows, rows - start)
        part = slice(start, start + n)
        h = hidden[part]
        ids = p(tgt.data_ptr() + 4 * step * start)
        code = L.ctb_ce_stats(_lib.ptr(h), _lib.ptr(head), n, vocab, d, ln(h.stride(0)), ln(head.stride(0)), ids, step,
                              p(work.pmax), p(work.psum), p(work.tlogit + 4 * start), None, ln(0), ln(0), ctypes.c_uint(0), None,
                              ln(0), ln(0), ctypes.c_uint(0), 0, 0, _lib.ptr(slab), ln(vocab), _lib.stream_ptr())
        _lib.check(code, "ctb_ce_stats")
        _combine(L, work, slabs, tgt, step, vocab, w, scale, device_scale, work.lse, work.coef, start, n)
        code = L.ctb_kept_logits_gradient(_lib.ptr(slab), ln(vocab), n, vocab, ids, step, p(work.lse + 4 * start),
                                          p(work.coef + 4 * start), _lib.stream_ptr())
        _lib.check(code, "ctb_kept_logits_gradient")
        g = slab.view(torch.bfloat16)[:n, :vocab]
        gemm(g, head, b_mn=True, out=dhidden[part])                                                    # dH = G @ W
        if need_dhead:
            gemm(g, h, a_mn=True, b_mn=True, out=dhead, accumulate=dhead_accumulate or start > 0)       # dW += G^T H
    return *_sums(L, work, rows), dhidden, dhead


def logits_ce_forward_backward(hidden, head, targets, weights, grad_scale: float = 1.0, *, chunk_rows: int = 4096,
                               need_dhead: bool = True, dhead_out: torch.Tensor | None = None,
                               dhead_accumulate: bool = False):
    """Cross-entropy through a materialised bf16 logits slab per row chunk (the ``pallas`` loss
    backend of the reference, src/causal_trainer/kernels/cross_entropy.py:216-251, 358-397):
    logits GEMM -> row statistics kernel -> dlogits written in place over the logits -> dH, dW.

    Returns ``(nll_sum, weight_sum, dhidden, dhead)``.  Rows with zero weight are skipped chunk-wise.
    """
    rows, d = hidden.shape
    vocab = head.shape[0]
    dev = hidden.device
    tgt = targets.to(torch.int32).contiguous()
    w = weights.to(torch.float32).contiguous()
    coef = w * grad_scale
    dhidden = torch.zeros_like(hidden)
    dhead = None
    if need_dhead:
        dhead = dhead_out if dhead_out is not None else torch.empty((vocab, d), dtype=torch.bfloat16, device=dev)
    chunk_rows = min(chunk_rows, rows)
    ldl = (vocab + 7) // 8 * 8
    slab = torch.empty((chunk_rows, ldl), dtype=torch.bfloat16, device=dev)
    lse = torch.empty(rows, dtype=torch.float32, device=dev)
    tl = torch.empty(rows, dtype=torch.float32, device=dev)
    L = _lib.lib()
    first = True
    for start in range(0, rows, chunk_rows):
        n = min(chunk_rows, rows - start)
        h = hidden[start:start + n]
        g = slab[:n, :vocab]
        gemm(h, head, out=g)
        code = L.ctb_logits_ce_stats(_lib.ptr(g), ctypes.c_long(ldl), n, vocab, _lib.ptr(tgt[start:start + n]),
                                     _lib.ptr(lse[start:start + n]), _lib.ptr(tl[start:start + n]), _lib.stream_ptr())
        _lib.check(code, "ctb_logits_ce_stats")
        code = L.ctb_logits_ce_backward(_lib.ptr(g), ctypes.c_long(ldl), n, vocab, _lib.ptr(tgt[start:start + n]),
                                        _lib.ptr(lse[start:start + n]), _lib.ptr(coef[start:start + n]),
                                        _lib.stream_ptr())
        _lib.check(code, "ctb_logits_ce_backward")
        gemm(g, head, b_mn=True, out=dhidden[start:start + n])
        if need_dhead:
            gemm(g, h, a_mn=True, b_mn=True, out=dhead, accumulate=(dhead_accumulate or not first))
        first = False
    nll = torch.where(w != 0, (lse - tl) * w, torch.zeros_like(lse))
    return nll.sum(), w.sum(), dhidden, dhead


class _CutCE(torch.autograd.Function):
    @staticmethod
    def forward(ctx, hidden, head, targets, weights, chunk_rows):
        nll, wsum, lse, coef = cut_ce_forward(hidden, head, targets, weights, 1.0)
        ctx.save_for_backward(hidden, head, targets, lse, coef)
        ctx.chunk_rows = chunk_rows
        return nll, wsum

    @staticmethod
    def backward(ctx, dnll, dw):
        hidden, head, targets, lse, coef = ctx.saved_tensors
        coef = coef * dnll.float()
        dh, dhead = cut_ce_backward(hidden, head, targets, lse, coef, chunk_rows=ctx.chunk_rows,
                                    need_dhead=ctx.needs_input_grad[1])
        return dh, dhead, None, None, None


def cut_cross_entropy(hidden, head, targets, weights, chunk_rows: int = 4096):
    """Differentiable projection-fused CE on the sm_100a kernels: (nll_sum, weight_sum)."""
    return _CutCE.apply(hidden, head, targets, weights, chunk_rows)
